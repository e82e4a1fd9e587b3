"""The warp-specialised CCF kernel at the edges of its particle streams,
reference pairs and shift groups (odd particle counts, work items of one and
of several particles, reference tiles with
one, two or three references, fewer shifts than a group, one shift group per
work item, both group sizes) against the general kernel, bit for bit: both run
the same sums in the same order."""
import numpy as np
import pytest

from gpuisac import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,NR,rng", [(1, 1, 5, 0.0), (1, 5, 29, 2.0), (2, 3, 7, 1.0), (3, 2, 29, 1.0), (9, 6, 12, 1.0),
                                        (17, 9, 30, 2.0), (8, 4, 1, 0.0), (7, 7, 37, 1.0), (10, 11, 45, 2.0),
                                        (1, 1300, 3, 0.0), (5, 700, 40, 0.0),
                                        # work items of 2, 8 (the last of one particle) and 4 particles
                                        (1301, 3, 5, 1.0), (1217, 14, 3, 1.0), (701, 13, 37, 0.0)])
def test_streams_equal_general_kernel(gpulib, cuda, monkeypatch, P, R, NR, rng):
    import torch
    from gpuisac.align import multi_ref_align_device
    D = max(40, 2 * NR + 6)
    st = synth.make_stack(P, D, min(R, 20), int(rng), 0.2, D * 0.4, 77 + P + R)
    refs = np.tile(st.refs, ((R + len(st.refs) - 1) // len(st.refs), 1, 1))[:R]
    refs = refs * (1.0 + 0.01 * np.arange(R, dtype=np.float32))[:, None, None]
    base = torch.from_numpy(np.random.default_rng(R).uniform(-1, 1, (P, 2)).astype(np.float32)).to(cuda)
    parts, refs = torch.from_numpy(st.particles).to(cuda), torch.from_numpy(np.ascontiguousarray(refs)).to(cuda)
    out = []
    for kernel in ("ws", "general"):
        monkeypatch.setenv("GPUISAC_CCF_KERNEL", kernel)
        out.append(multi_ref_align_device(parts, refs, NR, rng, rng, base_shifts=base, contraction_mode="fp32"))
    (d, p), (dg, pg) = out
    assert np.array_equal(d.cpu().numpy(), dg.cpu().numpy())
    assert np.array_equal(p.cpu().numpy(), pg.cpu().numpy())
