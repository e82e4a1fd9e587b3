"""The sampling offsets as the kernels form them (RingScale in
csrc/gpuisac_device.cuh): directions scaled in float and divided by the ring
count with Markstein's correction, against the oracle's template
(generate_polar_sampling_points, cuda/gpu_aln_common.cu:39-62) bit for bit."""
import numpy as np
import pytest

f32, f64 = np.float32, np.float64


def scaled(dirs, ring_num):
    """RingScale.offset for every ring, one float operation at a time (the two
    fused ones in double: e is exact there, q0 + e y rounds once more)"""
    n = f32(ring_num)
    y = f32(1.0) / n
    r = np.arange(1, ring_num + 1, dtype=f32)[:, None, None]
    m = (dirs[None] * r) * n
    q0 = m * y
    e = (m.astype(f64) - q0.astype(f64) * f64(n)).astype(f32)
    return (q0.astype(f64) + e.astype(f64) * f64(y)).astype(f32)


@pytest.mark.parametrize("ring_len", [256, 512])
def test_scaled_directions_are_the_template(oracle_mod, ring_len):
    dirs = oracle_mod.polar_template(1, ring_len)[0]  # one ring: the cosines and sines themselves
    for ring_num in range(1, 89):
        want = oracle_mod.polar_template(ring_num, ring_len)
        assert np.array_equal(scaled(dirs, ring_num), want), ring_num


def test_division_by_every_ring_count():
    """a seeded sample of 24-bit dividends for every ring count"""
    rng = np.random.default_rng(5)
    for ring_num in range(1, 89):
        m = (rng.integers(1 << 23, 1 << 24, 1 << 16) / f64(1 << 23)).astype(f32)
        n, y = f32(ring_num), f32(1.0) / f32(ring_num)
        q0 = m * y
        e = (m.astype(f64) - q0.astype(f64) * f64(n)).astype(f32)
        q = (q0.astype(f64) + e.astype(f64) * f64(y)).astype(f32)
        assert np.array_equal(q, m / n), ring_num
