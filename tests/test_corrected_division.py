"""The corrected quotients and reciprocals of the row kernels, in exact arithmetic: from an estimate of
20 bits, two Newton steps and one more give 1 / b rounded to nearest (unless every bit of b's
significand is set: the kernels then divide), and one remainder step a / b."""
from fractions import Fraction as F

import numpy as np
import pytest


def fma(a, b, c):
    return float(F(a) * F(b) + F(c))   # one rounding


def reciprocal(b, estimate):
    y = estimate
    for _ in range(3):
        y = fma(y, fma(-b, y, 1.0), y)
    return y


def significands(kind, rng):
    if kind == "random":
        return [int(x) for x in rng.integers(2**52, 2**53 - 1, 400)]
    if kind == "low":
        return [2**52 + k for k in range(40)]
    return [2**53 - 2 - k for k in range(40)]


@pytest.mark.parametrize("kind", ["random", "low", "high"])
def test_rounded_to_nearest(kind):
    rng = np.random.default_rng(3)
    for m in significands(kind, rng):
        b = float(m) * 2.0 ** int(rng.integers(-700, 600))
        for e in (-1.0, 0.0, 1.0, float(rng.uniform(-1, 1))):
            r = reciprocal(b, (1.0 / b) * (1.0 + e * 2.0**-20))
            assert r == 1.0 / b
        a = float(rng.integers(2**52, 2**53)) * 2.0 ** int(rng.integers(-150, 100))
        q = a * r
        assert fma(fma(-q, b, a), r, q) == a / b
