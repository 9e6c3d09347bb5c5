"""Elementwise assignments of single elements take four rows per thread: the
same values as numpy's at every remainder of rows, for strided, broadcast and
several operands and strided destinations."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "int8", "float64"])
@pytest.mark.parametrize("shape", [(3, 16, 7), (16, 2, 33), (17, 3, 5), (18, 40, 1001), (5, 19, 131), (35, 15, 9), (257, 64, 3)])
def test_odd_rows(shape, dtype):
    g = rng(shape[1])
    x = g.integers(-100, 100, shape).astype(dtype)
    y = g.integers(-9, 9, (1, shape[2])).astype(dtype)
    d, e = DeviceArray.from_numpy(x), DeviceArray.from_numpy(y)
    want = np.ascontiguousarray(x.transpose(1, 0, 2))
    out = DeviceArray.from_numpy(np.zeros_like(want))
    xg.assign(out, d.transpose((1, 0, 2)))
    np.testing.assert_array_equal(out.to_numpy(), want)
    rows = dtype != "float64" and shape[0] >= 16
    assert last_kernels()[0].endswith(", true>" if rows else "false>")
    out = DeviceArray.from_numpy(np.zeros((shape[1], shape[0], shape[2]), (x + y).dtype))
    xg.assign(out, d.transpose((1, 0, 2)) + e)
    np.testing.assert_array_equal(out.to_numpy(), want + y)
    # every second column, into rows apart
    wide = np.full((shape[1], shape[0], shape[2] + 3), 7, dtype)
    dst = DeviceArray.from_numpy(wide)
    xg.assign(dst[:, :, 1:1 + (shape[2] + 1) // 2], d.transpose((1, 0, 2))[:, :, ::2])
    wide[:, :, 1:1 + (shape[2] + 1) // 2] = want[:, :, ::2]
    np.testing.assert_array_equal(dst.to_numpy(), wide)
