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


@pytest.mark.parametrize("P,R,D", [
    (40, 2, 2), (40, 2, 9), (40, 3, 24), (64, 3, 48), (50, 2, 79), (50, 2, 80), (50, 2, 81), (50, 2, 82), (40, 2, 96),
    (40, 2, 112), (30, 2, 128), (20, 2, 129), (20, 2, 130), (20, 2, 144), (20, 2, 160), (12, 2, 162), (900, 1, 32),
])
def test_sums(gpulib, cuda, oracle_mod, P, R, D):
    """The sums alone at the sides where the sum kernel changes form: 80 / 81
    (rows a thread), 128 / 129 (passes), 160 / 162 and odd sides (global memory),
    multiples of 16 (rows staged apart), pieces of 2 members and of many.  The same
    bound: a source point in another cell than the restatement's is far outside."""
    from gpuisac.averages import class_averages
    imgs, peaks, bel = _case(P, R, D, 700 + D)
    out = class_averages(imgs, peaks, bel, 0.0, 0.2, False)
    _compare(oracle_mod, imgs, peaks, bel, 0.0, 0.2, False, out)


@pytest.mark.parametrize("D", [7, 48, 76, 100, 170])
def test_source_points_far_outside(gpulib, cuda, D):
    """A source point outside the image, infinite or NaN is the pixel itself."""
    from gpuisac.averages import class_averages
    rng = np.random.default_rng(D)
    imgs = rng.standard_normal((4, D, D)).astype(np.float32)
    peaks = np.zeros((4, 4, 4), np.float32)
    peaks[..., 1] = [1e30, -1e30, 3e6, np.nan]
    peaks[..., 2] = [-1e30, 9e6, 1e30, 0.0]
    out = class_averages(imgs, peaks, np.arange(4, dtype=np.int32), 0.0, 0.2, False)
    assert np.array_equal(out[0], imgs)
