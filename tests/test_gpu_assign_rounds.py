"""The group assignment's rounds in one launch (csrc/assign.cu) where it changes
form: more rounds than a launch runs (1,024), groups of 127 to 129 and 256 or 257
members (selection by counting or by digits, one to three digits), and the wide grid's first size (38,912
particles on 152 SMs).  The list equals the oracle's (integer work)."""
import numpy as np
import pytest

from test_gpu_assign import run_device, synth_peaks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref,nima,kind", [
    (1200, 2500, "dominant"),
    (3, 381, "classes"), (3, 384, "ties"), (3, 387, "signed"), (5, 1280, "dominant"), (5, 1289, "ties"),
    (20, 38912, "classes"), (20, 38911, "classes"),
])
def test_list_equals_oracle(oracle_mod, gpulib, cuda, nref, nima, kind):
    d = synth_peaks(nref, nima, nref + nima, kind)
    ids, _, rounds = run_device(d, cuda)
    assert rounds >= 1
    np.testing.assert_array_equal(ids, oracle_mod.assign_groups(d, nref, nima))


def test_more_rounds_than_a_launch(oracle_mod, gpulib, cuda):
    """Every particle ranks the groups alike: one group settles a round."""
    nref, nima = 1100, 2300
    d = np.random.default_rng(8).random((nref, nima), dtype=np.float32)
    d += 2.0 * np.arange(nref, 0, -1, dtype=np.float32)[:, None]
    ids, _, rounds = run_device(d, cuda)
    assert rounds >= nref
    np.testing.assert_array_equal(ids, oracle_mod.assign_groups(d, nref, nima))
