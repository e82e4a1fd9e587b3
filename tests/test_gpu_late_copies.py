"""The warp-specialised CCF kernel when its staging copies come too late: the
waits give up while the copies are in flight (gpuisac_test_late_ccf).  The
kernel lets them land before it reads the staging area or ends, hands over
every buffer to its FFT side, and the call reports the timeout; the next call
on the same context is right.  Item shapes on which the number of shift groups
after the wait that gave up is odd and even, of one and of several particles,
with one and with several references."""
import time

import numpy as np
import pytest

from gpuisac import GpuIsacError, synth

pytestmark = pytest.mark.gpu


# (40 rings: two shifts a group; 1,301 x 3: items of two particles)
@pytest.mark.parametrize("P,R,NR,rng", [(24, 6, 29, 2.0), (24, 6, 29, 1.0), (9, 1, 29, 2.0), (40, 5, 40, 1.0), (1301, 3, 5, 1.0)])
def test_late_copies_return_error_and_context_survives(gpulib, cuda, monkeypatch, P, R, NR, rng):
    import torch
    from gpuisac.align import multi_ref_align_device
    monkeypatch.setenv("GPUISAC_CCF_KERNEL", "ws")
    D = max(40, 2 * NR + 6)
    st = synth.make_stack(P, D, R, int(rng), 0.2, D * 0.4, 31)
    parts, refs = torch.from_numpy(st.particles).to(cuda), torch.from_numpy(st.refs).to(cuda)

    def run():
        return [t.cpu().numpy() for t in multi_ref_align_device(parts, refs, NR, rng, rng, contraction_mode="fp32")]

    want = run()
    gpulib.gpuisac_clear_error()
    gpulib.gpuisac_test_late_ccf(1)
    try:
        t0 = time.perf_counter()
        with pytest.raises(GpuIsacError, match="timed out"):
            run()
        assert time.perf_counter() - t0 < 10.0
    finally:
        gpulib.gpuisac_test_late_ccf(0)
        gpulib.gpuisac_clear_error()
    for w, g in zip(want, run()):
        assert np.array_equal(w, g)
