"""RingScale's division by the ring count (csrc/gpuisac_device.cuh) for every
24-bit dividend, with the device's roundings: q0 = RN(m y), e = RN(m - q0 N),
q = RN(q0 + e y) in one rounding, y = RN(1 / N), against the correctly rounded
m / N.  Odd counts up to the largest: a factor of two scales every step."""
import numpy as np
import pytest

f32, f64 = np.float32, np.float64


def fma_add(q0, e, y):
    """RN32(q0 + e y): the product is exact in 64 bits; where the 64-bit sum is a
    tie between two 32-bit numbers its own rounding error decides"""
    a, p = q0.astype(f64), e.astype(f64) * f64(y)
    s = a + p
    w = s - a
    lost = (a - (s - w)) + (p - w)
    tie = (s.view(np.int64) & ((1 << 29) - 1)) == 1 << 28
    s = np.where(tie & (lost != 0), np.nextafter(s, np.where(lost > 0, np.inf, -np.inf)), s)
    return s.astype(f32)


@pytest.mark.parametrize("first", range(1, 88, 8))
def test_every_dividend(first):
    for n in range(first, min(first + 8, 89), 2):
        y = f32(1.0) / f32(n)
        for lo in range(1 << 23, 1 << 24, 1 << 20):
            m = (np.arange(lo, lo + (1 << 20), dtype=f64) / f64(1 << 23)).astype(f32)
            q0 = m * y
            exact = m.astype(f64) - q0.astype(f64) * f64(n)
            e = exact.astype(f32)
            assert np.array_equal(e.astype(f64), exact)  # the remainder needs no rounding
            assert np.array_equal(fma_add(q0, e, y), m / f32(n)), n
