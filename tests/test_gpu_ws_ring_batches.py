"""The warp-specialised CCF kernel's references on their way to tensor memory, in
batches of five ring pairs per half of the contraction: ring counts around whole
and partial batches (2, 9 to 11, 18 to 22, 35 and 36 rings with four shifts per
group, 37 to 42 and 60 to 64 with two), full and partial reference tiles, against
the general kernel, bit for bit."""
import numpy as np
import pytest

from gpuisac import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NR", [2, 9, 10, 11, 18, 19, 20, 21, 22, 35, 36, 37, 39, 40, 41, 42, 60, 61, 63, 64])
def test_ring_batches_equal_general_kernel(gpulib, cuda, monkeypatch, NR):
    import torch
    from gpuisac.align import multi_ref_align_device
    D = max(40, 2 * NR + 6)
    st = synth.make_stack(5, D, 6, 1, 0.2, D * 0.4, 900 + NR)
    parts, refs = torch.from_numpy(st.particles).to(cuda), torch.from_numpy(st.refs).to(cuda)
    out = []
    for kernel in ("ws", "general"):
        monkeypatch.setenv("GPUISAC_CCF_KERNEL", kernel)
        out.append(multi_ref_align_device(parts, refs, NR, 1.0, 1.0, contraction_mode="fp32"))
    for a, b in zip(*out):
        assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())
