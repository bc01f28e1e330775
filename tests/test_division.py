"""The kernels' division by a launch-wide size (common.cuh div_by), restated in
exact rational arithmetic with its three FP32 roundings, against IEEE division."""

from fractions import Fraction

import numpy as np
import pytest


def rn32(x):
    """The FP32 value nearest to a rational, ties to even (normal range)."""
    if x == 0:
        return np.float32(0.0)
    near = np.float32(float(x))  # at most one step off
    best = None
    for c in (np.nextafter(near, np.float32(-np.inf)), near, np.nextafter(near, np.float32(np.inf))):
        d = abs(Fraction(float(c)) - x)
        even = int(np.float32(c).view(np.uint32)) & 1
        if best is None or (d, even) < best[0]:
            best = ((d, even), c)
    return np.float32(best[1])


def div_by(a, b):
    fa, fb = Fraction(float(a)), Fraction(float(b))
    rb = Fraction(float(np.float32(1.0) / b))
    q = Fraction(float(rn32(fa * rb)))
    rem = Fraction(float(rn32(fa - fb * q)))
    return rn32(rem * rb + q)


@pytest.mark.parametrize("size", [0.7, 0.9, 1.3, 0.91, 3.0, 0.1, 1.9999999, 1.0000001, 0.125, 37.5])
def test_rounds_as_the_division(size):
    b = np.float32(size)
    rng = np.random.default_rng(5)
    a = (rng.normal(size=400) * np.exp2(rng.uniform(-12, 12, 400))).astype(np.float32)
    ties = (b * rng.integers(1, 1 << 12, 100).astype(np.float32)).astype(np.float32)
    for x in np.concatenate([a, ties, -ties, [np.float32(0.0)]]):
        assert div_by(x, b) == x / b
