"""Scans along an axis of columns and of rows fold every element in order: the
same bits as a sequential fold, at the edges of the chunks (2 to 32 positions,
32 columns), of the groups of rows and of the rules that choose them."""
from __future__ import annotations

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

COLS = [(1, 5, 3), (4, 1, 7), (2, 4, 8), (3, 31, 65), (1, 32, 4), (1, 33, 100), (5, 64, 12), (7, 97, 1001), (1, 130, 4160),
        (16, 17, 1024), (1, 16, 16384), (3, 5, 131072), (1, 9, 131071), (1, 7, 524288), (2, 13, 262145)]
ROWS = [(1, 33), (31, 31), (32, 32), (33, 64), (100, 65), (4095, 257), (4096, 255), (4096, 257), (4097, 288), (4100, 289), (4111, 300)]


def check(x, axis, family):
    d = DeviceArray.from_numpy(x)
    want = np.cumsum(x, axis, dtype=x.dtype)
    got = ops.accumulate("cumsum", d, axis).to_numpy()
    assert last_kernels()[-1].startswith(family)
    np.testing.assert_array_equal(got, want)
    if x.dtype.kind == "f":
        # an expression of two operands
        e = DeviceArray.from_numpy(x[..., :1])
        got = ops.accumulate("cumsum", d + e, axis).to_numpy()
        np.testing.assert_array_equal(got, np.cumsum(x + x[..., :1], axis, dtype=x.dtype))
        y = x.copy()
        y[..., ::5] = np.nan
        got = ops.accumulate("nancumsum", DeviceArray.from_numpy(y), axis).to_numpy()
        np.testing.assert_array_equal(got, np.cumsum(np.nan_to_num(y), axis, dtype=x.dtype))
    np.testing.assert_array_equal(ops.accumulate("cumsum", d, axis, out=d).to_numpy(), want)


@pytest.mark.parametrize("dtype", ["float32", "float64", "int32"])
@pytest.mark.parametrize("shape", COLS)
def test_columns(shape, dtype):
    g = rng(shape[1])
    x = g.integers(-1000, 1001, shape) if dtype == "int32" else g.standard_normal(shape)
    check(x.astype(dtype), 1, "k_scan_col<")


@pytest.mark.parametrize("dtype", ["float32", "float64", "int32"])
@pytest.mark.parametrize("shape", ROWS)
def test_rows(shape, dtype):
    g = rng(shape[1])
    x = g.integers(-1000, 1001, shape) if dtype == "int32" else g.standard_normal(shape)
    x = x.astype(dtype)
    check(x, 1, "k_scan_rows<")
    # rows apart
    wide = np.zeros((shape[0], shape[1] + 3), dtype)
    wide[:, 1:1 + shape[1]] = x
    got = ops.accumulate("cumsum", DeviceArray.from_numpy(wide)[:, 1:1 + shape[1]], 1).to_numpy()
    np.testing.assert_array_equal(got, np.cumsum(x, 1, dtype=dtype))
