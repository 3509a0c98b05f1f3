"""The identities the fast forms of the march count loop rest on, in exact arithmetic on the CPU:
the scaled cell coordinate, its range, and the round-up division by two-part reciprocal."""
from fractions import Fraction

import numpy as np
import pytest

f32 = np.float32


def _round(x: Fraction) -> np.float32:
    """x > 0 to the nearest float32, ties to even."""
    e = 0
    while x >= 1 << 24:
        x, e = x / 2, e + 1
    while x < 1 << 23:
        x, e = x * 2, e - 1
    n, r = divmod(x.numerator, x.denominator)
    r = Fraction(r, x.denominator)
    n += r > Fraction(1, 2) or (r == Fraction(1, 2) and n & 1)
    return f32(np.ldexp(float(n), e))


@pytest.mark.parametrize("seed", [0, 1])
def test_round_up_division(seed):
    rng = np.random.default_rng(seed)
    for _ in range(60):
        b = f32(np.exp(rng.uniform(np.log(1e-6), np.log(10.0))))
        hi = f32(1.0) / b
        lo = f32(1.0 / float(b) - float(hi))
        B = Fraction(float(b))
        for a in [b, f32(2) * b, np.nextafter(b, f32(9)), np.nextafter(f32(3) * b, f32(0)),
                  *[f32(float(b) * k) for k in (3, 7, 511)], *f32(float(b) * np.exp(rng.uniform(0, 9, 20)))]:
            A = Fraction(float(a))
            q = _round(A * Fraction(float(hi)) + Fraction(float(a * lo)))
            if Fraction(float(q)) * B < A:
                q = np.nextafter(q, f32(np.inf))
            below = np.nextafter(q, f32(0))
            assert Fraction(float(q)) * B >= A > Fraction(float(below)) * B, (a, b)


@pytest.mark.parametrize("res", [16, 64, 128])
def test_scaled_coordinate(res):
    rng = np.random.default_rng(res)
    for _ in range(200):
        base = f32(np.exp(rng.uniform(np.log(1e-3), np.log(1e3)))) if rng.random() < 0.8 else f32(2.0 ** rng.integers(-4, 5))
        ils = f32(1.0) / base
        half = f32(0.5) * base
        x = np.concatenate([rng.uniform(-0.5, 0.5, 200).astype(f32) * base, [half, -half, f32(0), f32(1e-30),
                            np.nextafter(half, f32(0)), -np.nextafter(half, f32(0))]]).astype(f32)
        ref = ((x * ils).astype(f32) + f32(0.5)).astype(f32) * f32(res)
        s = ils * f32(res)
        got = ((x * s).astype(f32) + f32(res / 2)).astype(f32)
        np.testing.assert_array_equal(got, ref)
        assert got.min() >= 0 and got.max() <= res  # the cell needs only the clamp to R - 1
        if np.frexp(ils)[0] == 0.5:  # a power of two: the product is exact, one fused rounding is the same
            exact = x.astype(np.float64) * float(s) + res / 2
            np.testing.assert_array_equal(exact.astype(f32), ref)
