"""The tensor-core path at the edges of its FFT kernel's units (an even and an
odd number of shifts, one shift, several items per CTA) and of its particle
chunks (a second chunk, two reference tiles) against the FP32 path on the same
stacks, at the bar of the split tests: peaks within PEAK_RTOL (of at least 1 %
of the largest possible peak, the configuration tests' floor), the same tuples
on 99 %, the same best reference on 99.5 %."""
import numpy as np
import pytest

from gpuisac import synth

from test_gpu_align import ANGLE_TOL, PEAK_RTOL, circ_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,NR,rng", [(60, 9, 29, 1.5), (40, 11, 20, 1.0), (1300, 3, 7, 0.0), (700, 130, 12, 0.0),
                                        (30, 20, 29, 4.0)])
def test_units_and_chunks(gpulib, cuda, P, R, NR, rng):
    import torch

    from gpuisac import multi_ref_align_device
    D = 64
    st = synth.make_stack(P, D, R, int(rng), 0.2, D * 0.4, 930 + P)
    parts, refs = torch.from_numpy(st.particles).to(cuda), torch.from_numpy(st.refs).to(cuda)
    d32, p32 = (t.cpu().numpy() for t in multi_ref_align_device(parts, refs, NR, rng, rng, contraction_mode="fp32"))
    d16, p16 = (t.cpu().numpy() for t in multi_ref_align_device(parts, refs, NR, rng, rng, contraction_mode="bf16x3"))
    floor = 0.01 * 256.0 ** 2 * NR * (NR + 1) / 2
    assert (np.abs(d16.astype(np.float64) - d32) / np.maximum(np.abs(d32), floor)).max() <= PEAK_RTOL
    same = (p16[..., 1:] == p32[..., 1:]).all(-1) & (circ_diff(p16[..., 0], p32[..., 0]) < ANGLE_TOL)
    assert same.mean() >= 0.99, same.mean()
    assert (d16.argmax(0) == d32.argmax(0)).mean() >= 0.995
