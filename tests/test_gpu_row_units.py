"""Fused rows at the edges of their units: the bulk-copy form takes 32 / g rows
per warp (g = 4 .. 32 lanes), one row per block from 8 KiB on, and units that
start and end at any element.

Tolerance: that of the row normalisation tests (4e-6 / 1e-12 of the scale
(|x| + |mean|) / std for float32 / float64).
"""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300.device import DeviceArray

from util import assert_close_rel, rng

pytestmark = pytest.mark.gpu

REL = {"float32": 4e-6, "float64": 1e-12}


def normalize(view, out):
    xg.assign(out, (view - xg.rmean(view)) / xg.sqrt(xg.rvar(view) + 1e-5))
    return out.to_numpy().astype(np.float64)


def check(x, got, rel, what):
    xd = x.astype(np.float64)
    m = xd.mean(-1, keepdims=True)
    s = np.sqrt(xd.var(-1, keepdims=True) + 1e-5)
    assert_close_rel(got, (xd - m) / s, rel, (np.abs(xd) + np.abs(m)) / s, what)


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("cols", [1, 3, 4, 5, 16, 17, 51, 64, 65, 127, 128, 129, 256, 257, 511, 512, 513, 777, 1023,
                                  1025, 2047, 2049, 4095])
@pytest.mark.parametrize("rows", [203, 5003])  # one wave of warps, and more; no multiples of the rows per unit
def test_row_lengths(dt, cols, rows):
    g = rng(cols)
    flat = g.standard_normal(rows * cols + 8).astype(dt)
    d = DeviceArray.from_numpy(flat)
    for off in (0, 1, 3):  # rows from every phase of a 16-byte granule
        v = d[off:off + rows * cols].reshape((rows, cols))
        x = flat[off:off + rows * cols].reshape(rows, cols)
        check(x, normalize(v, DeviceArray.empty((rows, cols), dt)), REL[dt], f"{cols} at {off}")


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("cols", [33, 64, 301, 1500, 2050])
def test_rows_of_a_view_and_two_leaves(dt, cols):
    """Rows at a distance (one row per warp), a second leaf with its own phase
    and a strided destination; nothing outside the destination is written."""
    g = rng(cols)
    x = g.standard_normal((37, cols + 5)).astype(dt)
    w = g.standard_normal((37, cols)).astype(dt)
    d, dw = DeviceArray.from_numpy(x)[:, 2:cols + 2], DeviceArray.from_numpy(w)
    out = DeviceArray.from_numpy(np.full((37, cols + 3), 7.0, dt))
    o = out[:, 1:cols + 1]
    xg.assign(o, (d - xg.rmean(d)) / xg.sqrt(xg.rvar(d) + 1e-5) + dw)
    got = out.to_numpy()
    assert (got[:, 0] == 7).all() and (got[:, cols + 1:] == 7).all()
    xd = x[:, 2:cols + 2].astype(np.float64)
    m, s = xd.mean(-1, keepdims=True), np.sqrt(xd.var(-1, keepdims=True) + 1e-5)
    assert_close_rel(got[:, 1:cols + 1].astype(np.float64), (xd - m) / s + w, REL[dt], (np.abs(xd) + np.abs(m)) / s + np.abs(w),
                     "two leaves")


@pytest.mark.parametrize("cols", [7, 50, 100, 200, 2051])
def test_special_rows_beside_plain_ones(cols):
    """float64 rows with an infinity or NaN take the FP64 path; the rows that
    share their warp keep the fixed-point results, bit for bit."""
    g = rng(cols)
    x = g.standard_normal((5003, cols))
    y = x.copy()
    y[::3, cols // 2] = np.inf
    y[1::9, 0] = np.nan
    ref = normalize(DeviceArray.from_numpy(x), DeviceArray.empty(x.shape, "float64"))
    with np.errstate(invalid="ignore"):
        got = normalize(DeviceArray.from_numpy(y), DeviceArray.empty(x.shape, "float64"))
    plain = np.isfinite(y).all(1)
    np.testing.assert_array_equal(got[plain], ref[plain])
    assert np.isnan(got[np.isnan(y).any(1)]).all()
