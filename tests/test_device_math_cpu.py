"""Float sequences of rcv_device.cuh that stand in for slower ones on the
device, restated in numpy over every argument they can have.

A fused multiply-add of float32 values is a float64 sum of an exact product
(24 + 24 bits) rounded to float32; where the sum itself has to round to float64
first, the second rounding can differ where the float64 sum falls on a tie: those
cases are taken again in rational numbers."""
from fractions import Fraction

import numpy as np
import pytest

f32, f64 = np.float32, np.float64


def rounded(x):
    """Float32 nearest to a Fraction in the normal range, ties to even."""
    e = 0
    while abs(x) < Fraction(2) ** e:
        e -= 1
    while abs(x) >= Fraction(2) ** (e + 1):
        e += 1
    n = x / Fraction(2) ** (e - 23)
    whole = n.numerator // n.denominator
    rest = n - whole
    return f32(float((whole + (rest > Fraction(1, 2) or (rest == Fraction(1, 2) and whole % 2 == 1))) * Fraction(2) ** (e - 23)))


def fma(a, b, c):
    product = a.astype(f64) * b.astype(f64)
    total = product + c.astype(f64)
    out = total.astype(f32)
    lost = (total - c.astype(f64)) != product  # the float64 sum rounded
    tie = (total.view(np.uint64) & np.uint64((1 << 29) - 1)) == np.uint64(1 << 28)
    for i in np.nonzero(lost & tie)[0]:
        out[i] = rounded(Fraction(float(a[i])) * Fraction(float(b[i])) + Fraction(float(c[i])))
    return out


@pytest.mark.parametrize("ulps", [-1, 0, 1, 2])
def test_log_quotient_is_the_division_for_every_argument(ulps):
    """(m - 1) / (m + 1) for all 1 - u, u = k 2^-23 (every value next1d gives),
    from a hardware reciprocal up to two ulps off the rounded one."""
    x = (1.0 - np.arange(1 << 23, dtype=f64) * 2.0 ** -23).astype(f32)
    bits = x.view(np.uint32)
    m = np.unique(((bits & np.uint32(0x007FFFFF)) | np.uint32(0x3F800000))).view(f32)
    m = np.where(m > f32(1.41421356237), m * f32(0.5), m)
    a, b = m - f32(1), m + f32(1)
    y = (f32(1) / b).astype(f32)
    y = (y.view(np.int32) + np.int32(ulps)).view(f32)
    y = fma(fma(-b, y, np.ones_like(b)), y, y)
    y[b == f32(1.99999988)] = f32(0.50000006)
    q = (a * y).astype(f32)
    s = fma(fma(-b, q, a), y, q)
    assert np.array_equal(s, (a / b).astype(f32))


@pytest.mark.parametrize("D", [1, 2, 3, 17, 64, 255, 1000, 65537, (1 << 21) - 1])
def test_axis_by_directed_rounding_matches_floor(D):
    """floor(g) and the weight from g + 1.5 * 2^23 rounded towards minus
    infinity, for points in and a little outside the unit interval, at voxel
    centres and their neighbours."""
    rng = np.random.default_rng(D)
    p = np.concatenate([rng.random(200_000), [0.0, 1.0, -1e-6, 1.0 + 1e-6, -1e-3, 1.001, 1e-30, 0.5 / D],
                        (rng.integers(0, D, 5000) + 0.5) / D]).astype(f32)
    p = np.concatenate([p, np.nextafter(p, f32(2)), np.nextafter(p, f32(-1))])
    g = fma(p, np.full_like(p, D), np.full_like(p, -0.5))
    # the sum rounded down: float64 holds it exactly (|g| < 2^22, 24-bit significand at 2^-149 and up aside)
    t = np.floor(g.astype(f64)) + 12582912.0
    t = t.astype(f32)
    assert np.array_equal(t.astype(f64), np.floor(g.astype(f64)) + 12582912.0)  # whole numbers below 2^24
    fl = t - f32(12582912.0)
    cell = np.clip(t.view(np.int32).astype(np.int64) - 0x4B3FFFFF, 0, D)
    old_fl = np.floor(g)
    old = np.clip(np.clip(old_fl, -1, D).astype(np.int64) + 1, 0, D)
    assert np.array_equal(fl, old_fl) and np.array_equal(cell, old)
