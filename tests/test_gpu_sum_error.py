"""Rounding error of float64 row reductions against 64 bits: rms over 16384
rows no larger than that of the order in which 32 lanes share a row (lane i
vectors i, i + 32, ... in turn, then halves of the warp), restated here.

The errors of two orders on the same rows are nearly independent, so the ratio
of their rms over N rows has a standard deviation of about sqrt(2 / N) = 1.1%
(1.6% for errors of twice a normal kurtosis): a ratio up to 1.05 is equality.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

N = 16384


def lanes(x, vec):
    """x as (lane, step, row, element of the vector), absent ones NaN."""
    n = x.shape[1]
    steps = -(-n // (32 * vec))
    y = np.full((x.shape[0], steps * 32 * vec), np.nan)
    y[:, :n] = x
    return y.reshape(x.shape[0], steps, 32, vec).transpose(2, 1, 0, 3)


def halves(a):
    while a.shape[0] > 1:
        a = a[:a.shape[0] // 2] + a[a.shape[0] // 2:]
    return a[0]


def chain(x, vec, square):
    y = lanes(x, vec)
    s = np.zeros((32, x.shape[0]))
    for k in range(y.shape[1]):
        for j in range(vec):
            d = y[:, k, :, j]
            if square:  # fma: one rounding
                t = (d.astype(np.longdouble) * d + s).astype(np.float64)
            else:
                t = s + d
            s = np.where(np.isnan(d), s, t)
    return halves(s)


def rms(e):
    return math.sqrt(float(np.mean(np.square(e.astype(np.float64)))))


@pytest.mark.parametrize("cols", [32, 48, 63, 64, 128, 180, 255, 256, 512])
@pytest.mark.parametrize("op", ["sum", "mean", "variance", "norm_sq"])
def test_rows(op, cols):
    g = rng(cols)
    x = g.standard_normal((N, cols)) + 0.25
    vec = 2 if cols % 2 == 0 else 1
    L = x.astype(np.longdouble)
    if op in ("sum", "mean"):
        want, ref = L.sum(1), chain(x, vec, False)
        if op == "mean":  # (its division rounds too)
            want, ref = want / cols, ref / cols
        ref = ref - want
    elif op == "norm_sq":
        want = np.square(L).sum(1)
        ref = chain(x, vec, True) - want
    else:
        m = L.mean(1, keepdims=True)
        want = np.square(L - m).mean(1)
        d = x - x[:, :1]
        s1, s2 = chain(d, vec, False), chain(d, vec, True)
        ref = (s2 - s1 * (s1 / cols)) / cols - want
    got = ops.reduce(op, DeviceArray.from_numpy(x), [1]).to_numpy()
    assert rms(got - want) <= 1.05 * rms(ref), (rms(got - want), rms(ref))


def test_unaligned_rows():
    """Rows of 32 at an odd element: single elements, as at 33."""
    x = rng(7).standard_normal((N, 32)) + 0.25
    d = DeviceArray.from_numpy(np.concatenate([[0.0], x.ravel()]))[1:].reshape((N, 32))
    want = x.astype(np.longdouble).sum(1)
    assert rms(ops.reduce("sum", d, [1]).to_numpy() - want) <= 1.05 * rms(chain(x, 1, False) - want)
