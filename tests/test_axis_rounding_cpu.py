"""axis_coord_magic (rcv_device.cuh) against axis_coord, restated in numpy: cell
and interpolation weight from the sum g + 1.5 * 2^23 rounded towards minus
infinity, the rounding taken from the exact sum."""
import numpy as np
import pytest

f32, f64 = np.float32, np.float64
MAGIC = f32(12582912.0)


def points(D):
    rng = np.random.default_rng(D)
    p = np.concatenate([rng.random(100_000), [0.0, 1.0, -1e-6, 1.0 + 1e-6, -1e-3, 1.001, 1e-30, 0.5 / D],
                        (rng.integers(0, D, 5000) + 0.5) / D]).astype(f32)
    return np.concatenate([p, np.nextafter(p, f32(2)), np.nextafter(p, f32(-1))])


def scaled(p, D):
    """fmaf(p, D, -0.5): a float64 product is exact, and the sum's float64 rounding
    leaves 29 bits beyond the float32 result (both roundings: the points of
    test_device_math_cpu.py, which takes the ties in rational numbers)."""
    return (p.astype(f64) * f64(D) - 0.5).astype(f32)


def add(g, mode):
    """g + MAGIC in float32, rounded down or to nearest, from the exact sum s + err (TwoSum)."""
    a, b = g.astype(f64), f64(MAGIC)
    s = a + b
    bb = s - a
    err = (a - (s - bb)) + (b - bb)
    r = s.astype(f32)
    above = (r.astype(f64) > s) | ((r.astype(f64) == s) & (err < 0))
    return np.where(above, np.nextafter(r, f32(-np.inf)), r) if mode == "down" else r


def magic(g, D, mode="down", offset=0x4B3FFFFF):
    t = add(g, mode)
    weight = g - (t - MAGIC)
    cell = np.clip(t.view(np.int32).astype(np.int64) - offset, 0, D)
    return cell, weight


def plain(g, D):
    fl = np.floor(g)
    return np.clip(np.clip(fl, -1, D).astype(np.int64) + 1, 0, D), g - fl


@pytest.mark.parametrize("D", [1, 2, 3, 17, 64, 255, 1000, 65537, (1 << 21) - 1])
def test_cell_and_weight(D):
    g = scaled(points(D), D)
    for got, want in zip(magic(g, D), plain(g, D)):
        assert np.array_equal(got, want)


def test_a_mistake_would_be_seen():
    """Rounding to nearest or another offset gives other cells and weights."""
    g = scaled(points(64), 64)
    cell, weight = plain(g, 64)
    near = magic(g, 64, mode="nearest")
    assert np.mean(near[0] != cell) > 0.3 and np.mean(near[1] != weight) > 0.3
    assert np.mean(magic(g, 64, offset=0x4B400000)[0] != cell) > 0.9
