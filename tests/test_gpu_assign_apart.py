"""The group assignment's two forms (csrc/assign.cu: rounds in one cooperative
grid, or each step a launch of its own) on both sides of the line between them
(400,000 particles; 36,000,000 pairs with more than 1,000 groups; 22,000,000
with 2,000 groups and more tiles of 32 particles than the grid has CTAs): the
form is the one the size asks for and the list equals the oracle's (integer
work)."""
import numpy as np
import pytest

from gpuisac import GpuIsacError

from test_gpu_assign import run_device, synth_peaks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref,nima,kind,apart", [
    (4, 400_000, "classes", False), (4, 400_001, "classes", True), (3, 400_003, "ties", True), (7, 400_010, "signed", True),
    (1, 400_001, "ties", True), (40, 400_039, "dominant", True),
    (1001, 35_964, "classes", False), (1001, 35_965, "classes", True),
    (2000, 11_000, "classes", False), (2000, 11_001, "ties", True),
])
def test_form_and_list(oracle_mod, gpulib, cuda, nref, nima, kind, apart):
    d = synth_peaks(nref, nima, nref + nima, kind)
    before = gpulib.gpuisac_launch_count()
    ids, bel, rounds = run_device(d, cuda)
    launches = gpulib.gpuisac_launch_count() - before
    assert launches == (4 * rounds + 3 if apart else 1)
    np.testing.assert_array_equal(ids, oracle_mod.assign_groups(d, nref, nima))
    maxasi = nima // nref
    want = np.repeat(np.arange(nref), maxasi)
    np.testing.assert_array_equal(bel[ids[:nref * maxasi]], want)
    assert (bel[ids[nref * maxasi:nima]] == ids[-1]).all()


def test_nan_is_refused(gpulib, cuda):
    import torch
    from gpuisac.assign import assign_groups_device
    d = torch.rand(2, 400_001, device=cuda)
    d[1, 77] = float("nan")
    with pytest.raises(GpuIsacError, match="NaN"):
        assign_groups_device(d)
    gpulib.gpuisac_clear_error()
    d[1, 77] = 0.5
    ids, bel, _ = assign_groups_device(d, with_id_list=False)
    assert ids is None and int((bel == 0).sum()) in (200_000, 200_001)
