"""The division by a launch constant of the reductions' finishers (`div_by` in
csrc/xtg_device.cuh), restated step for step with exact arithmetic: a r, two
remainders and two corrections equal the IEEE quotient for every count that a
mean or variance divides by (a reciprocal rounded to nearest, 1 .. 2^40)."""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np
import pytest


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # rounded once, to nearest even


def div_by(a, b):
    r = 1.0 / b
    q = a * r
    eq, ea = math.frexp(q)[1] + 1022, math.frexp(a)[1] + 1022
    if not (128 <= eq < 1920 and 128 <= ea < 1920):
        return a / b
    q = fma(fma(-q, b, a), r, q)
    return fma(fma(-q, b, a), r, q)


@pytest.mark.parametrize("seed", range(4))
def test_quotients_are_correctly_rounded(seed):
    g = np.random.default_rng(seed)
    counts = [float(n) for n in [*range(1, 40), 2**16 - 1, 2**28, 2**28 + 3, 2**40 - 1,
                                 *g.integers(3, 2**40, 60), *(2.0 ** g.integers(1, 40, 20) - 1)]]
    for b in counts:
        for a in [*g.standard_normal(20), *(g.standard_normal(10) * np.exp2(g.integers(-1000, 1000, 10))),
                  b * (1 + 2.0**-52), b * 3.0, -b / 3.0, float(np.nextafter(b * 7, 0))]:
            assert div_by(float(a), b) == float(a) / b, (a, b)
