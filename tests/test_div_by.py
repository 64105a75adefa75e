"""div_by (device_common.cuh): quotients of one divisor by its reciprocal and
two fused corrections round correctly.  The steps are restated in exact
rational arithmetic, each result rounded once (float of a Fraction rounds to
nearest, ties to even), and compared with the rounded quotient."""
import random
from fractions import Fraction

import pytest


def rn(x: Fraction) -> float:
    return x.numerator / x.denominator


def fma(a, b, c):
    return rn(Fraction(a) * Fraction(b) + Fraction(c))


def div_by(a, b):
    y = 1.0 / b
    q0 = a * y
    q1 = fma(fma(-q0, b, a), y, q0)
    return fma(fma(-q1, b, a), y, q1)


@pytest.mark.parametrize("seed", range(4))
def test_random(seed):
    rng = random.Random(seed)
    for _ in range(4000):
        a = rng.uniform(-1, 1) * 2.0 ** rng.randint(-60, 60)
        b = rng.uniform(1, 2) * 2.0 ** rng.randint(-30, 30)
        assert div_by(a, b) == a / b


def test_extreme_mantissas():
    ends = [1.0, 1.0 + 2.0 ** -52, 1.0 + 2.0 ** -51, 1.5, 2.0 - 2.0 ** -52, 2.0 - 2.0 ** -51, 1.0 + 2.0 ** -26,
            2.0 - 2.0 ** -26, 4.0 / 3.0, 5.0 / 3.0, 2.0 ** 0.5]
    for a in ends:
        for b in ends:
            for s in (1.0, 8.0, 2.0 ** -40):
                assert div_by(a * s, b) == (a * s) / b
    s = float((1 << 53) - 1)  # the Monte Carlo draws' divisor
    for a in (0.0, 1.0, 2.0, s - 1.0, s, float(1 << 52), float((1 << 52) + 1)):
        assert div_by(a, s) == a / s
