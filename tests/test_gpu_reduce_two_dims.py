"""Reductions over dims that do not collapse, with fewer lanes than a warp per
output: integers, maxima and their NaN order exact, float32 sums within 2^-23
|exact| + 2^-36 sum|x|, float64 within 1e-13 sum|x|."""
from __future__ import annotations

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

SHAPES = [(3, 5000, 7), (2, 9001, 16), (5, 140000, 3), (2, 4097, 100), (20, 4500, 7), (3, 8200, 33), (7, 20, 5)]


@pytest.mark.parametrize("shape", SHAPES)
def test_axes_0_and_2(shape):
    g = rng(shape[1])
    x = g.integers(-1000, 1001, shape).astype("int32")
    d = DeviceArray.from_numpy(x)
    np.testing.assert_array_equal(ops.reduce("sum", d, [0, 2]).to_numpy(), x.sum((0, 2)))
    assert last_kernels()[0].startswith("k_reduce_row<")
    np.testing.assert_array_equal(ops.reduce("amax", d, [0, 2]).to_numpy(), x.max((0, 2)))
    x = g.standard_normal(shape) * 10.0 ** g.integers(-2, 3, shape)
    for dt in ("float32", "float64"):
        h = x.astype(dt)
        w = h.astype(np.longdouble)
        d = DeviceArray.from_numpy(h)
        exact, mag = w.sum((0, 2)), np.abs(w).sum((0, 2))
        tol = 2.0**-23 * np.abs(exact) + 2.0**-36 * mag if dt == "float32" else 1e-13 * mag
        assert (np.abs(ops.reduce("sum", d, [0, 2]).to_numpy() - exact) <= tol).all()
        np.testing.assert_array_equal(ops.reduce("amin", d, [0, 2]).to_numpy(), h.min((0, 2)))
        # NaNs as the sequential fold takes them: m = m > x ? m : x in order
        h[0, :: max(1, shape[1] // 50), shape[2] // 2] = np.nan
        h[0, 1, 0] = np.nan
        m = h[0, :, 0].copy()
        with np.errstate(invalid="ignore"):
            for i in range(shape[0]):
                for k in range(shape[2]):
                    if i or k:
                        m = np.where(m > h[i, :, k], m, h[i, :, k])
        np.testing.assert_array_equal(ops.reduce("amax", DeviceArray.from_numpy(h), [0, 2]).to_numpy(), m)
