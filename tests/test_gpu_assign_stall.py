"""The group assignment's grid barrier when it runs out: every CTA gives up its
bounded wait and returns, the call reports the timeout at once, and the next
call on the same context is right (grids of one, a few and two or four CTAs per
SM; with and without the list)."""
import time

import numpy as np
import pytest

from gpuisac import GpuIsacError
from gpuisac.assign import assign_groups_device

from test_gpu_assign import run_device, synth_peaks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref,nima,with_list", [(1, 9, True), (7, 300, True), (200, 4099, False), (200, 20000, True),
                                                 (5, 40000, True)])
def test_stalled_barrier_returns_error_and_context_survives(gpulib, cuda, oracle_mod, nref, nima, with_list):
    import torch
    d = synth_peaks(nref, nima, 3)
    dev = torch.from_numpy(d).to(cuda)
    gpulib.gpuisac_clear_error()
    gpulib.gpuisac_test_stall_ccf(64)
    try:
        t0 = time.perf_counter()
        with pytest.raises(GpuIsacError, match="timed out"):
            assign_groups_device(dev, with_id_list=with_list)
        assert time.perf_counter() - t0 < 10.0
    finally:
        gpulib.gpuisac_test_stall_ccf(0)
        gpulib.gpuisac_clear_error()
    ids, _, _ = run_device(d, cuda)
    np.testing.assert_array_equal(ids, oracle_mod.assign_groups(d, nref, nima))
