"""The Monte Carlo kernels' uniform draw: v / (2^53 - 1) for an integer v < 2^53
is the number after v 2^-53 (kernels_mc.cu, xorshift64), and 0 for v = 0."""
import math
import random

import pytest

MAX = float(2 ** 53 - 1)


def draw(v):
    return math.nextafter(math.ldexp(float(v), -53), 2.0) if v else 0.0


@pytest.mark.parametrize("seed", range(4))
def test_random(seed):
    rng = random.Random(seed)
    for _ in range(20000):
        v = rng.getrandbits(rng.randint(1, 53))
        assert draw(v) == float(v) / MAX


def test_ends():
    for b in range(54):
        for d in range(-3, 4):
            v = (1 << b) + d
            if 0 <= v < 1 << 53:
                assert draw(v) == float(v) / MAX
