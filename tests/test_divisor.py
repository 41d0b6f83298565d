"""The FP64 sweeps' division by a launch constant (one multiplication and two
fused multiply-adds, stencil.cuh div_by) returns the correctly rounded
quotient: checked in exact rational arithmetic."""
import random
from fractions import Fraction

import pytest


def _fma(a: float, b: float, c: float) -> float:
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # rounded once


def _div_by(x: float, d: float) -> float:
    r = 1.0 / d
    q = x * r
    return _fma(_fma(-q, d, x), r, q)


# the divisors of a run: dx^2 of the lattice sizes, scale factors
DIVISORS = [(20.0 / N) ** 2 for N in (8, 48, 64, 100, 256, 512)] + [1.0, 1.0000244, 1.7, 18.25, 0.37]


@pytest.mark.parametrize("d", DIVISORS)
def test_division_by_a_constant_is_correctly_rounded(d):
    rng = random.Random(int(d * 1e6))
    for _ in range(3000):
        # mantissas near 1, near 2 and anywhere, over the magnitudes of fields and Laplacians
        m = rng.choice((1.0 + rng.randint(0, 8) * 2.0 ** -52, 2.0 - rng.randint(1, 8) * 2.0 ** -53, rng.uniform(1, 2)))
        x = rng.choice((-1, 1)) * m * 2.0 ** rng.randint(-90, 20)
        assert _div_by(x, d) == x / d, (x, d)
    assert _div_by(0.0, d) == 0.0
