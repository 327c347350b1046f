"""Division by a small integer as the wall function does it (d3q19.cuh: div_small): p y with y the
correctly rounded reciprocal, corrected once by fused multiply-adds, is the correctly rounded p / n."""
from fractions import Fraction

import numpy as np


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))      # exact, rounded once


def test_corrected_product_is_the_quotient():
    rng = np.random.default_rng(0)
    p = np.ldexp(rng.uniform(-1, 1, 60), rng.integers(-40, 3, 60))
    p = np.concatenate([p, [0.1, 1 / 3, np.nextafter(1.0, 0), np.nextafter(75.0, 100)]])
    for n in range(1, 76):
        y = 1.0 / n
        for v in map(float, p):
            q = v * y
            assert fma(fma(-q, float(n), v), y, q) == v / n, (v, n)
