"""The averages' row and column passes (csrc/averages.cu) at the image sides where
their tiles end: the smallest and largest side, one more and one less than whole
row tiles (16) and column tiles (8 of the half spectrum), odd sides (no D / 2
term), and more groups than the half spectra held at once (415 of side 200).
Averages within 2e-5 of the largest average value of the FP64 restatement, the
bound of the other averaging tests: FP32 sums of at most 256 terms."""
import numpy as np
import pytest

from test_gpu_averages import _case, _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,D,fl,ff,center", [
    (12, 2, 2, 0.2, 0.2, True), (12, 2, 3, 0.2, 0.2, True), (20, 3, 14, 0.3, 0.1, True), (20, 3, 15, 0.3, 0.1, False),
    (20, 3, 16, 0.2, 0.0, True), (20, 3, 17, 0.0, 0.2, True), (20, 3, 33, 0.2, 0.2, True), (20, 3, 94, 0.2, 0.2, True),
    (20, 3, 127, 0.3, 0.2, True), (9, 2, 161, 0.2, 0.2, True), (6, 2, 255, 0.2, 0.2, True), (6, 2, 256, 0.4, 0.1, True),
    (440, 430, 200, 0.2, 0.2, True),
])
def test_sides(gpulib, cuda, oracle_mod, P, R, D, fl, ff, center):
    from gpuisac.averages import class_averages
    imgs, peaks, bel = _case(P, R, D, 300 + D)
    out = class_averages(imgs, peaks, bel, fl, ff, center)
    assert np.isfinite(out[0]).all()
    _compare(oracle_mod, imgs, peaks, bel, fl, ff, center, out)
