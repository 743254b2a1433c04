"""The quotient that box numbers and interpolation weights are made of (grid_geom.cuh, divide): two Newton-Raphson steps on
a * (1 / b) round to the float that a division gives."""
from fractions import Fraction

import numpy as np
import pytest


def to_float(v):
    """A fraction rounded once to a (normal) float: to the nearest, ties to even."""
    if v == 0:
        return np.float32(0.0)
    e = 0
    m = abs(v)
    while m >= 1 << 24:
        m /= 2
        e += 1
    while m < 1 << 23:
        m *= 2
        e -= 1
    whole, rest = divmod(m, 1)
    whole = int(whole) + (1 if rest > Fraction(1, 2) or (rest == Fraction(1, 2) and int(whole) & 1) else 0)
    return np.float32(float(np.ldexp(float(whole), e)) * (1 if v > 0 else -1))


def fma(a, b, c):
    return to_float(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c)))


def divide(a, b, r):
    q = to_float(Fraction(float(a)) * Fraction(float(r)))
    q = fma(fma(-q, b, a), r, q)
    return fma(fma(-q, b, a), r, q)


def weight_divisors():
    """The denominators of the Lagrange weights, as make_interp_consts forms them."""
    f = np.float32
    h = f(1) / f(3)
    sp = [h / f(2)]
    for _ in range(2):
        sp.append(sp[-1] + h)
    den = []
    for i in range(3):
        d = f(1)
        for j in range(3):
            if i != j:
                d = f(d * f(sp[i] - sp[j]))
        den.append(d)
    return den


@pytest.mark.parametrize("kind", ["weights", "boxes"])
def test_quotient_is_the_divisions(kind):
    rng = np.random.default_rng(3)
    if kind == "weights":
        cases = [(np.float32(v), d) for d in weight_divisors() for v in np.concatenate([rng.uniform(-1, 1, 150), 2.0 ** rng.uniform(-50, 0, 50)])]
    else:      # widths between 1e-20 and 1e20, the mantissas for which a reciprocal is least exact among them
        widths = np.concatenate([10.0 ** rng.uniform(-19.5, 19.5, 300), np.ldexp(2.0 - 2.0 ** -23 * rng.integers(1, 4, 100), rng.integers(-20, 20, 100))])
        cases = [(np.float32(np.float32(w) * rng.uniform(0, 130.001)), np.float32(w)) for w in widths]
    for a, b in cases:
        assert divide(a, b, np.float32(1) / b) == np.float32(a / b), (a, b)
