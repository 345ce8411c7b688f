"""The quotient by a constant of the density kernels (div_const in
mph_device.cuh): a first product with the rounded reciprocal and two residual
corrections.  Its operations, each rounded once, in exact rational arithmetic
against the correctly rounded quotient: the same bits."""
import random
from fractions import Fraction

import pytest


def fma(a: float, b: float, c: float) -> float:
    return float(Fraction(a) * Fraction(b) + Fraction(c))   # one rounding, to nearest even


def div_const(a: float, c: float, y: float) -> float:
    q = a * y
    q = fma(fma(-q, c, a), y, q)
    return fma(fma(-q, c, a), y, q)


# radii and R2g of particle spacings from 0.1 mm to 1 m, and divisors next to a power of two
CONSTANTS = [3.5 * 0.005, 1.7 * 0.005, 3.5 * 0.01, 1.7 * 0.01, 3.1 * 1e-4, 2.1, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52, 1.0, 4.2e-7]


@pytest.mark.parametrize("c", CONSTANTS)
def test_quotient_bits(c):
    rng = random.Random(5)
    y = 1.0 / c
    for k in range(4000):
        a = (1.0 + rng.random()) * 2.0 ** rng.randint(-60, 20) * rng.choice((-1.0, 1.0))
        if k < 40:
            a = c * (1.0 + (k - 20) * 2.0 ** -52) * (k % 3 + 1)   # quotients next to whole numbers
        assert div_const(a, c, y) == a / c, (a, c)
    assert div_const(0.0, c, y) == 0.0
