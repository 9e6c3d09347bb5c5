"""Column reductions over rows that vectors do not divide: lane-strided
outputs at the edges of a warp's 32 or 64 columns and of a batch of 8 rows,
splits, several kept and reduced dims, a broadcast leaf.

Tolerances: selections, positions and integers exact against the oracle;
float32 sums within 1e-6 of sum|x|, float64 within 1e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray, HostArray

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["float32", "float64", "int32", "int16"])
@pytest.mark.parametrize("shape", [(3, 7, 33), (5, 8, 63), (2, 9, 65), (1, 641, 129), (4, 1, 1001), (9, 300, 35)])
def test_columns(dt, shape):
    g = rng(sum(shape))
    x = (g.integers(-50, 50, shape) * (1 if dt.startswith("int") else 0.5)).astype(dt)
    if dt.startswith("float"):
        x[0, 0, ::5] = np.nan  # the first elements of some columns
        x[-1, -1, 1::7] = np.inf
    d = DeviceArray.from_numpy(x)
    for op in ("argmax", "argmin"):
        np.testing.assert_array_equal(ops.argreduce(op, d, 1).to_numpy(), O.argreduce(op, HostArray(x), 1))
    for axes in ([1], [0, 1], [0]):
        y = np.nan_to_num(x, nan=0.5, posinf=3.0).astype(dt)
        dy, b = DeviceArray.from_numpy(y), g.integers(1, 4, (shape[0], 1, 1)).astype(dt)
        db = DeviceArray.from_numpy(b)
        for op in ("amax", "amin"):
            np.testing.assert_array_equal(ops.reduce(op, dy, axes).to_numpy(), O.reduce(op, HostArray(y), axes))
        got = ops.reduce("sum", dy * db, axes).to_numpy()
        if dt.startswith("int"):
            np.testing.assert_array_equal(got, O.reduce("sum", HostArray(y) * HostArray(b), axes))
        else:
            e = y.astype(np.float64) * b
            tol = 1e-6 if dt == "float32" else 1e-12
            assert (np.abs(got - e.sum(tuple(axes))) <= tol * np.abs(e).sum(tuple(axes))).all()
