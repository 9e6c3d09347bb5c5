"""The segmented scan's whole-line copies, folds and stores at the edges of its
tiles (512 elements) and segments: integers exact, float32 within the
double-float bound of the exact prefix (2^-23 |exact| + 2^-36 sum|x|), float64
within 1e-12 of the prefix magnitude; the same in place."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

SHAPES = [(1, 4), (1, 508), (1, 512), (1, 516), (3, 1020), (2, 1536 + 8), (5, 512 * 37 + 12), (1, 4864 * 512 - 4),
          (1, 4864 * 512 * 2 + 516), (7, 100_004), (1, 511), (2, 1023)]


@pytest.fixture(autouse=True)
def segments():
    xg.set_option("scan.strategy", 2)
    yield
    xg.set_option("scan.strategy", -1)


@pytest.mark.parametrize("shape", SHAPES)
def test_segmented_scans(shape):
    g = rng(shape[0] * 1000 + shape[1])
    for dt in ("int32", "int64", "int16"):
        x = g.integers(-1000, 1001, shape).astype(dt)
        d = DeviceArray.from_numpy(x)
        got = ops.accumulate("cumsum", d, 1)
        assert last_kernels()[-1].startswith("k_scan_seg_apply")
        np.testing.assert_array_equal(got.to_numpy(), np.cumsum(x, 1, dtype=got.to_numpy().dtype))
        if dt != "int16":
            np.testing.assert_array_equal(ops.accumulate("cumsum", d, 1, out=d).to_numpy(), np.cumsum(x, 1, dtype=dt))
    x = g.standard_normal(shape)
    x[:, : shape[1] // 2] *= 1e3
    for dt in ("float32", "float64"):
        h = x.astype(dt)
        w = h.astype(np.longdouble)
        exact, mag = np.cumsum(w, 1), np.cumsum(np.abs(w), 1)
        tol = 2.0**-23 * np.abs(exact) + 2.0**-36 * mag if dt == "float32" else 1e-12 * mag
        d = DeviceArray.from_numpy(h)
        a = ops.accumulate("cumsum", d, 1).to_numpy()
        assert (np.abs(a - exact) <= tol).all()
        assert ops.accumulate("cumsum", d, 1, out=d).to_numpy().tobytes() == a.tobytes()
        # an expression: the register form
        d = DeviceArray.from_numpy(h)
        assert (np.abs(ops.accumulate("cumsum", d + d, 1).to_numpy() - 2 * exact) <= 2 * tol).all()
