"""Rounding error of a float32 row's variance in fused rows, against 64 bits:
rms over 16384 rows no larger than with the row shared by 32 lanes (256 above
512 single elements), each lane's squared deviations in four float32 chains and
the lanes' sums compensated, restated here.

Two orders' errors on the same rows are nearly independent, so the ratio of
their rms has a standard deviation of about sqrt(2 / N) = 1.1%; pairs of squares
instead of single ones add up to 2% at 27 elements: the bound is 1.06.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

N = 16384
F = np.float32


def fma(a, b, c):
    return (a.astype(np.float64) * b + c).astype(F)


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def shared_by(x, mean, lanes, vec):
    """Sum of squared deviations of every row."""
    n = x.shape[1]
    steps = -(-n // (lanes * vec))
    d = np.full((N, steps * lanes * vec), np.nan, F)
    d[:, :n] = x - mean
    d = d.reshape(N, steps, lanes, vec).transpose(2, 1, 3, 0)
    chains = [np.zeros((lanes, N), F) for _ in range(4)]
    for i in range(steps * vec):
        v = d[:, i // vec, i % vec]
        chains[i % 4] = np.where(np.isnan(v), chains[i % 4], fma(v, v, chains[i % 4]))
    hi = (chains[0] + chains[1]) + (chains[2] + chains[3])
    lo = np.zeros_like(hi)
    while hi.shape[0] > 1:
        h = hi.shape[0] // 2
        s, e = two_sum(hi[:h], hi[h:])
        lo = (lo[:h] + lo[h:]) + e
        hi = s
    return hi[0] + lo[0]


def rms(e):
    return math.sqrt(float(np.mean(np.square(e.astype(np.float64)))))


@pytest.mark.parametrize("cols", [27, 51, 64, 99, 131, 191, 255, 321, 777])
def test_variance(cols):
    x = rng(cols).standard_normal((N, cols)).astype(F)
    L = x.astype(np.longdouble)
    want = np.square(L - L.mean(1, keepdims=True)).mean(1)
    mean = (x.astype(np.float64).sum(1).astype(F) / F(cols))[:, None]
    vec = 4 if cols % 4 == 0 else 1
    ref = shared_by(x, mean, 32 if cols <= 512 * vec else 256, vec) / F(cols)
    d = DeviceArray.from_numpy(x)
    out = DeviceArray.empty(x.shape, "float32")
    xg.assign(out, d * xg.scalar(0, "float32") + xg.rvar(d))
    got = out.to_numpy()[:, 0]
    new, old = rms((got - want) / want), rms((ref - want) / want)
    assert new <= 1.06 * old, (new, old)
