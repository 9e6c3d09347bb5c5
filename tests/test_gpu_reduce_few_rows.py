"""Column reductions of few rows that vectors do not divide: every number of rows
behind the batches of eight, four and two.

Tolerances: integers, selections and positions exact against the oracle; float32
sums within 1e-6 of sum|x|, float64 within 1e-12 (those of the reduction tests).
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray, HostArray

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["float32", "float64", "uint8", "int16"])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 6, 7, 8, 9, 13, 15, 16, 23])
def test_columns(rows, dt):
    g = rng(rows)
    x = g.integers(0, 9, (rows, 1001)).astype(dt) if dt in ("uint8", "int16") else g.standard_normal((rows, 1001)).astype(dt)
    d, h = DeviceArray.from_numpy(x), HostArray(x)
    for op in ("amax", "amin"):
        np.testing.assert_array_equal(ops.reduce(op, d, [0]).to_numpy(), O.reduce(op, h, [0]))
        np.testing.assert_array_equal(ops.argreduce("arg" + op[1:], d, 0).to_numpy(), O.argreduce("arg" + op[1:], h, 0))
    s = ops.reduce("sum", d, [0]).to_numpy()
    if dt in ("uint8", "int16"):
        np.testing.assert_array_equal(s, x.sum(0, dtype=s.dtype))
        return
    X = x.astype(np.longdouble)
    rel = 1e-6 if dt == "float32" else 1e-12
    assert (np.abs(s - X.sum(0)) <= rel * np.abs(X).sum(0)).all()
    assert (np.abs(ops.reduce("norm_sq", d, [0]).to_numpy() - np.square(X).sum(0)) <= rel * np.square(X).sum(0)).all()
    v = np.square(X - X.mean(0)).mean(0)
    assert (np.abs(ops.reduce("variance", d, [0]).to_numpy() - v) <= rel * np.square(X - X[0]).mean(0) + 1e-300).all()
