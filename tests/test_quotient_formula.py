"""The red-black stopping test divides by a float as a product with its
correctly rounded reciprocal and one correction (fl_multigrid.cu, over_scale);
restated here with exact rationals, each operation rounded once, and checked
against the division."""
from fractions import Fraction

import numpy as np


def quotient(x, scale, rcp):
    q = x * rcp
    rem = float(Fraction(x) - Fraction(q) * Fraction(scale))  # an FMA: one rounding
    return float(Fraction(rem) * Fraction(rcp) + Fraction(q))


def test_corrected_product_equals_the_division():
    rng = np.random.default_rng(3)
    n = 4000
    scale = np.abs(rng.standard_normal(n)) * 2.0 ** rng.integers(-60, 60, n)
    scale[::9] = 2.0 ** rng.integers(-149, 127, scale[::9].size)
    scale[::11] = np.nextafter(np.float32(2.0) ** rng.integers(-20, 20, scale[::11].size).astype(np.float32), np.float32(0))
    scale[:3] = np.finfo(np.float32).max, np.finfo(np.float32).tiny, 2.0 ** -149
    scale = scale.astype(np.float32).astype(np.float64)
    # count * p - sum: floats, and their differences in double
    a = (rng.standard_normal(n) * 2.0 ** rng.integers(-60, 60, n)).astype(np.float32).astype(np.float64)
    b = (a * (1 + rng.integers(-3, 4, n) * 2.0 ** -23)).astype(np.float32).astype(np.float64)
    x = rng.integers(1, 5, n) * a - np.where(rng.random(n) < 0.7, b, 0.0)
    for xv, s in zip(x.tolist(), scale.tolist()):
        assert quotient(xv, s, 1.0 / s) == xv / s, (xv, s)
