"""The column solves divide by table entries through their reciprocals (step_kernels.cuh:div_by): q = a r, q + r (a - q d) with
r = 1/d, all rounded to nearest.  Restated here in exact rationals and compared with the division itself."""
import random
from fractions import Fraction

import pytest


def div_by(a, d, r):
    q = a * r
    res = float(Fraction(a) - Fraction(q) * Fraction(d))       # fma(-q, d, a)
    return float(Fraction(q) + Fraction(res) * Fraction(r))    # fma(res, r, q)


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e150])
def test_quotients_are_the_correctly_rounded_ones(scale):
    rng = random.Random(int(scale % 1000) + 3)
    for _ in range(4000):
        d = -rng.uniform(1.0, 2.0) * 2.0 ** rng.randint(-20, 20)
        a = rng.uniform(-1.0, 1.0) * 10.0 ** rng.randint(-6, 6) * scale
        assert div_by(a, d, 1.0 / d) == a / d


@pytest.mark.parametrize("d", [-1.0, -0.25, -2.0 ** 40, -(2.0 - 2.0 ** -52), -(1.0 + 2.0 ** -52)])
@pytest.mark.parametrize("a", [0.0, 1.0, 2.0 - 2.0 ** -52, -(1.0 + 2.0 ** -52), 3.0])
def test_edges(a, d):
    assert div_by(a, d, 1.0 / d) == a / d
