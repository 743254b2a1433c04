"""The double reciprocal that the kernel's grid values are made of (convolve.cu, kernel_value): two Newton-Raphson steps from a
float reciprocal are as exact as a division.  The steps square the error of the start (below 2^-21) to 2^-84, so only the
last rounding is left: half a unit of the last place and 2^-31 of one, and the double that a division gives unless 1 / t
lies that close to a tie (t one unit below a power of two, for one)."""
import math
from fractions import Fraction

import numpy as np


def fma(a, b, c):
    """a * b + c rounded once (the quotient of Python's integers is)."""
    v = Fraction(a) * Fraction(b) + Fraction(c)
    return v.numerator / v.denominator


def test_two_steps_from_a_float_reciprocal():
    rng = np.random.default_rng(1)
    t = np.concatenate([1.0 + rng.random(4000), 1.0 + rng.random(1000) * 2.0 ** -40, 10.0 ** rng.uniform(0, 37, 4000),
                        2.0 ** rng.integers(0, 122, 500) * (1 + 2.0 ** -52 * rng.integers(0, 3, 500)), 2.0 ** rng.integers(1, 122, 500) - 1])
    for x in t:
        x = float(x)
        exact = float(np.float32(1) / np.float32(x))
        for ulps in (-2, 0, 2):                               # CUDA's fast division is within two units of the last place
            r = exact * (1 + ulps * 2.0 ** -23)
            r1 = fma(r, fma(-x, r, 1.0), r)
            r2 = fma(r1, fma(-x, r1, 1.0), r1)
            off = abs(Fraction(r2) - 1 / Fraction(x)) / Fraction(math.ulp(1.0 / x))
            assert off <= Fraction(1, 2) + Fraction(1, 2 ** 31)
            assert r2 == 1.0 / x or off >= Fraction(1, 2)
            assert np.float32(r2) == np.float32(1.0 / x)


def test_values_beyond_the_range_of_floats():
    """From 1e37 on the steps run on t 2^-160 and the result is scaled back: a float's zero or subnormal, as by division."""
    rng = np.random.default_rng(2)
    for x in np.concatenate([10.0 ** rng.uniform(37, 78, 2000), [1.0000001e37, 8.5e37, 1.7e38, 3.5e38, 1.4e45, 2.9e45, 1e78]]):
        t = float(x) * 2.0 ** -160
        assert 2.0 ** -126 < t < 2.0 ** 126                   # the divisors for which CUDA's fast division is within two units
        exact = float(np.float32(1) / np.float32(t))
        for ulps in (-2, 0, 2):
            r = exact * (1 + ulps * 2.0 ** -23)
            r1 = fma(r, fma(-t, r, 1.0), r)
            r2 = fma(r1, fma(-t, r1, 1.0), r1)
            assert np.float32(r2 * 2.0 ** -160) == np.float32(1.0 / float(x))
