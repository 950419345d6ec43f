"""The quotient n/Frund of the quantised velocity correction by Markstein's correction step on the
rounded reciprocal equals the IEEE quotient: float-valued Frund, integers n up to 2^31, in exact
rational arithmetic (``float(Fraction)`` rounds correctly, as the FMA does)."""
from fractions import Fraction

import numpy as np
import pytest


def markstein(n, b):
    y = 1.0 / b
    q0 = n * y
    r = Fraction(n) - Fraction(q0) * Fraction(b)
    assert Fraction(float(r)) == r                      # the FMA's remainder is exact
    return float(Fraction(q0) + r * Fraction(y))


@pytest.mark.parametrize("seed", range(4))
def test_markstein_quotient_is_the_ieee_quotient(seed):
    rng = np.random.default_rng(seed)
    for _ in range(1500):
        top = np.float32(10.0 ** rng.uniform(-2, 3))
        b = float(np.float32(rng.choice([8000.0, 10000.0])) / top)
        for n in (float(rng.integers(1, 1 << 31)), float(rng.integers(1, 1 << 12)), float((1 << 31) - 1 - rng.integers(0, 9)),
                  -float(rng.integers(1, 1 << 31)), float(1 << 31), 1.0):
            assert markstein(n, b) == n / b, (n, b)
    # divisors with the longest and the shortest float significands
    for b in (float(np.float32(16777215.0 / 2048)), 8192.0, float(np.nextafter(np.float32(8192), np.float32(0)))):
        for n in rng.integers(1, 1 << 31, 500):
            assert markstein(float(n), b) == float(n) / b
