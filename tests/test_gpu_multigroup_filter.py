"""The stability test's average filter (csrc/multigroup.cu) at sides where its CTAs
of 256 values end inside a row, at a whole number of rows or with one value left
(16, 17, 32, 45, 90, 100), one average and several, against the FP64 restatement
within the bound of the other filter test."""
import numpy as np
import pytest

from test_gpu_multigroup import FILTER_RTOL, Session, class_stack, close_images

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,R", [(16, 1), (17, 3), (32, 2), (45, 5), (90, 2), (100, 3)])
def test_filter_sides(gpulib, cuda, oracle_mod, D, R):
    parts, cid = class_stack(6 * R, D, R, 40 + D)
    s = Session(parts, cid, max(3, D // 2 - 5), 1.0)
    try:
        before = s.averages()
        s.filter(0.2, 0.2)
        after = s.averages()
    finally:
        s.close()
    assert np.isfinite(after).all()
    close_images(after, oracle_mod.tanl_filter_averages(before, 0.2, 0.2), FILTER_RTOL)
