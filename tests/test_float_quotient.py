"""The quotient that box numbers and interpolation weights are made of (grid_geom.cuh, divide): two Newton-Raphson steps on
a * (1 / b) round to the float that a division gives.  First the method, in fractions; then the charges that the device
makes of it, against divisions on the host."""
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


# widths of a map: divisions as the compiler has them below 1e-20 and above 1e20 for a box of 130, the quotient in between
@pytest.mark.gpu
@pytest.mark.parametrize("width", [1e-22, 1e-16, 1e-3, 1.0, 37.7, 1e5, 1e18, 1e23])
@pytest.mark.parametrize("centre", [0.0, 0.4, -3.0])
def test_charges_are_those_of_divisions(engine, width, centre):
    """A point alone in its box leaves its nine weights on the grid: box and weights bit for bit, for points on box borders, next
    to them, and anywhere."""
    f, boxes = np.float32, 130
    rng = np.random.default_rng(8)
    lo, hi = f((centre - 0.5) * width), f((centre + 0.5) * width)
    bw = f((hi - lo) / f(boxes))
    border = np.arange(1, boxes, dtype=np.float32) * bw + lo
    axis = np.concatenate([border, np.nextafter(border, f(np.inf)), np.nextafter(border, f(-np.inf)), rng.uniform(lo, hi, 400).astype(f)])
    axis = axis[(axis > lo) & (axis < hi)]

    def weights(c):
        box = np.clip(((c - lo) / bw).astype(np.int64), 0, boxes - 1)
        lower = (box.astype(np.longdouble) * np.longdouble(bw) + np.longdouble(lo)).astype(f)     # one rounding, as a fused operation has
        inside = (c - lower) / bw
        h = f(1) / f(3)
        sp = [h / f(2)]
        for _ in range(2):
            sp.append(sp[-1] + h)
        L = []
        for j, den in enumerate(weight_divisors()):
            v = np.ones_like(c)
            for k in range(3):
                if k != j:
                    v = v * (inside - sp[k])
            L.append(v / den)
        return box, np.stack(L)

    x, y = rng.permutation(np.repeat(axis, 6)), rng.permutation(np.repeat(axis, 6))
    x[:2], y[:2] = (lo, hi), (hi, lo)
    bx, Lx = weights(x)
    by, Ly = weights(y)
    box = bx * boxes + by
    alone = np.bincount(box, minlength=boxes * boxes)[box] == 1
    assert alone.sum() > 1000
    with np.errstate(over="ignore", invalid="ignore"):
        w = engine.repulsive(np.stack([x, y]), True)[2]
    for a in range(3):
        for b in range(3):
            assert np.array_equal(w[bx[alone] * 3 + a, by[alone] * 3 + b, 0], (Lx[a] * Ly[b])[alone])
