"""Row reductions over units: many short rows, rows that start at any element,
1 .. 32 lanes per row, the first and last unit of an array, leaves beside the
streamed one.

Tolerances: integers, selections and positions bit-exact against the oracle;
float32 sums within 1e-6 of sum|x|, float64 within 1e-12, variances relative
1e-6 / 1e-12 of the FP64 value (those of the reduction tests).
"""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from oracle import oracle as O
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray, HostArray

from util import rng

pytestmark = pytest.mark.gpu

COLS = [2, 3, 4, 5, 8, 16, 17, 24, 31, 32, 33, 63, 64, 65, 128, 255, 256, 257, 511, 513, 1023, 1024]


def data(g, n, dt):
    if dt.startswith("int"):
        return g.integers(-1000, 1001, n).astype(dt)
    return g.standard_normal(n).astype(dt)


def close(got, want, scale, dt, what):
    rel = 1e-12 if dt == "float64" else 1e-6
    np.testing.assert_array_less(np.abs(got - want), rel * scale + 1e-300, err_msg=what)


@pytest.mark.parametrize("dt", ["float32", "float64", "int32"])
@pytest.mark.parametrize("cols", COLS)
def test_rows(dt, cols):
    g = rng(cols)
    rows = 4101  # past the bound from which units are used, no multiple of the rows per unit
    flat = data(g, rows * cols + 8, dt)
    d = DeviceArray.from_numpy(flat)
    for off in (0, 1, 3):
        v = d[off:off + rows * cols].reshape((rows, cols))
        x = np.ascontiguousarray(flat[off:off + rows * cols].reshape(rows, cols))
        what = f"{dt} {cols} at {off}"
        xd = x.astype(np.float64)
        for op in ("amax", "amin"):
            np.testing.assert_array_equal(ops.reduce(op, v, [1]).to_numpy(), O.reduce(op, HostArray(x), [1]), err_msg=what)
        np.testing.assert_array_equal(ops.argreduce("argmax", v, 1).to_numpy(), O.argreduce("argmax", HostArray(x), 1),
                                      err_msg=what)
        s = ops.reduce("sum", v, [1]).to_numpy()
        if dt == "int32":
            np.testing.assert_array_equal(s, x.sum(1, dtype=np.int32), err_msg=what)
            continue
        close(s, xd.sum(1), np.abs(xd).sum(1), dt, what)
        var = xd.var(1)
        close(ops.reduce("variance", v, [1]).to_numpy(), var, var + 1e-12 * (xd * xd).mean(1), dt, what)


@pytest.mark.parametrize("cols", [4, 15, 64, 301])
def test_leaves_beside_the_streamed_ones(cols):
    """A vector broadcast over the rows, a value per row, a second streamed
    leaf at another phase; the fused store equals the two calls bit for bit."""
    g = rng(cols)
    rows = 5000
    a, w = (g.standard_normal(rows * cols + 4).astype(np.float32) for _ in range(2))
    b, r = g.standard_normal(cols).astype(np.float32), g.standard_normal((rows, 1)).astype(np.float32)
    da, dw = (DeviceArray.from_numpy(t)[k:k + rows * cols].reshape((rows, cols)) for t, k in ((a, 0), (w, 3)))
    e = da * DeviceArray.from_numpy(b) + dw * DeviceArray.from_numpy(r)
    A, W = (t[k:k + rows * cols].reshape(rows, cols).astype(np.float64) for t, k in ((a, 0), (w, 3)))
    close(ops.reduce("sum", e, [1]).to_numpy(), (A * b + W * r).sum(1), (np.abs(A * b) + np.abs(W * r)).sum(1), "float32", "sum")
    E1, E2 = (DeviceArray.empty((rows, cols), "float32") for _ in range(2))
    r1 = ops.assign_reduce(E1, e, "sum", axes=[1])
    xg.assign(E2, e)
    r2 = ops.reduce("sum", E2, [1])
    np.testing.assert_array_equal(E1.to_numpy(), E2.to_numpy())
    np.testing.assert_array_equal(r1.to_numpy(), r2.to_numpy())


@pytest.mark.parametrize("dt", ["float32", "float64"])
def test_special_values_and_strided_rows(dt):
    """NaNs, infinities and signed zeros in some of a warp's rows; rows at a
    distance (not streamed), a strided result."""
    g = rng(5)
    x = g.integers(-2, 3, (4200, 21)).astype(dt) * np.array(0.5, dt)
    x[::7, 4] = np.nan
    x[3::11, 0] = np.nan
    x[5::13, 8] = np.inf
    x[6::5, :] = 0.0
    x[6::5, 3] = -0.0
    d = DeviceArray.from_numpy(x)
    for op in ("amax", "amin"):
        got, want = ops.reduce(op, d, [1]).to_numpy(), O.reduce(op, HostArray(x), [1])
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(np.signbit(got[~np.isnan(got)]), np.signbit(want[~np.isnan(want)]))
    np.testing.assert_array_equal(ops.argreduce("argmax", d, 1).to_numpy(), O.argreduce("argmax", HostArray(x), 1))
    y = np.ascontiguousarray(x[:, 2:17])
    out = DeviceArray.from_numpy(np.full(8400, 9.0, dt))
    ops.reduce("amin", d[:, 2:17], [1], out=out[::2])
    got = out.to_numpy()
    assert (got[1::2] == 9).all()
    np.testing.assert_array_equal(got[::2], O.reduce("amin", HostArray(y), [1]))
