"""Transposes at the edges of full tiles (64 and 32 wide) and in tiles of
other extents (small ones, several planes per tile), one and two operands, destinations
of several strides: the same values as numpy's."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

SHAPES = [(3, 64, 64), (3, 63, 65), (2, 128, 130), (1, 129, 200), (5, 127, 33), (700, 22, 36), (3001, 3, 5), (4, 2, 9000),
          (2, 9001, 3), (300, 1, 70), (7, 70, 75), (40, 300, 40), (1000, 17, 64), (9, 66, 257), (2, 33, 1000)]


@pytest.mark.parametrize("dtype", ["float32", "float64", "int8"])
@pytest.mark.parametrize("shape", SHAPES)
def test_transposes(shape, dtype):
    g = rng(shape[1])
    x = g.integers(-100, 100, shape).astype(dtype)
    y = g.integers(-9, 9, (shape[0], 1, shape[2])).astype(dtype)
    d, e = DeviceArray.from_numpy(x), DeviceArray.from_numpy(y)
    for perm in ((2, 0, 1), (2, 1, 0), (1, 0, 2), (0, 2, 1), (1, 2, 0)):
        want = np.ascontiguousarray(x.transpose(perm))
        out = DeviceArray.from_numpy(np.zeros_like(want))
        xg.assign(out, d.transpose(perm))
        np.testing.assert_array_equal(out.to_numpy(), want)
        # two operands, one of them broadcast
        w = (x + y).transpose(perm)
        out = DeviceArray.from_numpy(np.zeros(w.shape, w.dtype))
        xg.assign(out, d.transpose(perm) + e.transpose(perm))
        np.testing.assert_array_equal(out.to_numpy(), w)
        # a destination with rows apart
        wide = np.full(want.shape[:2] + (want.shape[2] + 3,), 7, dtype)
        dst = DeviceArray.from_numpy(wide)
        xg.assign(dst[:, :, 1:1 + want.shape[2]], d.transpose(perm))
        wide[:, :, 1:1 + want.shape[2]] = want
        np.testing.assert_array_equal(dst.to_numpy(), wide)


def test_the_tiles_are_used():
    x = DeviceArray.from_numpy(np.zeros((2, 128, 190), "float32"))
    xg.assign(DeviceArray.from_numpy(np.zeros((2, 190, 128), "float32")), x.transpose((0, 2, 1)))
    assert last_kernels()[0].startswith("k_transpose<") and last_kernels()[0].endswith(", 64, 64, 1, 4>")
    x = DeviceArray.from_numpy(np.zeros((700, 22, 36), "float32"))
    xg.assign(DeviceArray.from_numpy(np.zeros((700, 36, 22), "float32")), x.transpose((0, 2, 1)))
    assert last_kernels()[0].startswith("k_transpose<") and last_kernels()[0].endswith(", 16, 32, 8, 4>")
