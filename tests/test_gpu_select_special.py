"""amax / amin / argmax / argmin of rows with infinities and NaNs, rows of 21 to 5000 elements:
values and signs of zeros against the oracle's fold in order (a NaN is replaced
by what follows it, the last of equal values wins), and such rows at a cost of
the same order as plain ones."""
from __future__ import annotations

import time

import numpy as np
import pytest

from oracle import oracle as O
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray, HostArray, device_sync

from util import rng

pytestmark = pytest.mark.gpu


def special_rows(g, rows, cols, dt):
    x = (g.integers(-3, 4, (rows, cols)) * 0.5).astype(dt)
    r = np.arange(rows)
    kind = r % 12
    x[kind == 0, g.integers(0, cols)] = np.nan
    x[kind == 1, -1] = np.nan                      # the fold ends on it
    x[kind == 2, 0] = np.nan
    x[kind == 3] = np.nan
    x[kind == 4, g.integers(0, cols)] = -np.inf
    x[kind == 5, g.integers(0, cols)] = np.inf
    x[kind == 6] = -np.inf
    x[kind == 7, : cols // 2] = np.nan
    x[kind == 7, cols // 2:] = -np.inf             # nothing but an end behind the last NaN
    x[kind == 8] = np.where(g.random((int((kind == 8).sum()), cols)) < 0.5, 0.0, -0.0)
    x[kind == 8, cols // 3] = np.nan
    x[kind == 9] = np.inf
    x[kind == 9, cols // 4] = np.nan
    x[kind == 10, cols - 2] = np.nan
    x[r % 24 == 11] = -np.inf                      # NaNs before the first of equal ends
    x[r % 24 == 11, : cols // 5] = np.nan
    x[r % 24 == 23] = np.inf
    x[r % 24 == 23, 1] = np.nan
    return x


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("rows,cols", [(4104, 21), (4104, 64), (4104, 301), (4101, 1024), (40, 33), (40, 301), (36, 4096), (13, 5000)])
def test_values(rows, cols, dt):
    x = special_rows(rng(cols), rows, cols, dt)
    flat = np.concatenate([np.zeros(1, dt), x.ravel()])
    d = DeviceArray.from_numpy(flat)[1:].reshape((rows, cols))
    for a in (DeviceArray.from_numpy(x), d):
        for op in ("amax", "amin"):
            got, want = ops.reduce(op, a, [1]).to_numpy(), O.reduce(op, HostArray(x), [1])
            if rows < 100 and cols > 1000:  # several work items per row: NaNs of several items meet in no set order
                n = ~np.isnan(x).any(1)
                got, want = got[n], want[n]
            np.testing.assert_array_equal(got, want, err_msg=op)
            n = ~np.isnan(want)
            np.testing.assert_array_equal(np.signbit(got[n]), np.signbit(want[n]), err_msg=op)
            got, want = ops.argreduce("arg" + op[1:], a, 1).to_numpy(), O.argreduce("arg" + op[1:], HostArray(x), 1)
            np.testing.assert_array_equal(got, want, err_msg="arg" + op[1:])


@pytest.mark.parametrize("axes,shape", [([0, 2], (7, 500, 40)), ([1], (300, 70, 5))])
def test_other_axes(axes, shape):
    g = rng(2)
    x = special_rows(g, shape[0] * shape[1], shape[2], "float64").reshape(shape)
    for op in ("amax", "amin"):
        got, want = ops.reduce(op, DeviceArray.from_numpy(x), axes).to_numpy(), O.reduce(op, HostArray(x), axes)
        assert got.shape == want.shape
        n = ~np.isnan(x).any(axis=tuple(axes))  # (NaNs of several runs meet in no set order)
        np.testing.assert_array_equal(got[n], want[n])


@pytest.mark.parametrize("dt", ["float32", "float64"])
@pytest.mark.parametrize("rows,cols", [(4104, 5), (1500, 9), (4104, 21), (4104, 64), (4101, 301), (40, 33), (40, 301), (4101, 1024)])
@pytest.mark.parametrize("form", ["dense", "strided", "in place"])
def test_fused_with_the_assignment(form, rows, cols, dt):
    """Stored and reduced in one call: the same as assigned and then reduced."""
    x = special_rows(rng(cols), rows, cols, dt)
    d = DeviceArray.from_numpy(x)
    for op in ("amax", "amin"):
        if form == "in place":
            d = out = DeviceArray.from_numpy(x)
        elif form == "dense":
            out = DeviceArray.empty((rows, cols), dt)
        else:
            out = DeviceArray.from_numpy(np.zeros((rows, cols + 3), dt))[:, 1:cols + 1]
        r = ops.assign_reduce(out, d + d, op, axes=[1]).to_numpy()
        got, want = out.to_numpy(), O.reduce(op, HostArray(x + x), [1])
        np.testing.assert_array_equal(got, x + x)
        np.testing.assert_array_equal(r, want, err_msg=op)
        np.testing.assert_array_equal(r, ops.reduce(op, out, [1]).to_numpy())
        n = ~np.isnan(want)
        np.testing.assert_array_equal(np.signbit(r[n]), np.signbit(want[n]), err_msg=op)


@pytest.mark.parametrize("dt,special", [("float64", -np.inf), ("float64", np.nan), ("float32", np.nan)])
def test_cost(dt, special):
    """One special value per row of 1024: three passes over a cached row where
    plain rows take one, so a factor of ten is far above what it may cost (a
    lane that walks the row alone takes 25 times a plain row's time)."""
    x = rng(1).standard_normal((16384, 1024)).astype(dt)
    y = x.copy()
    y[np.arange(16384), np.arange(16384) % 1024] = special
    best = []
    for a in (DeviceArray.from_numpy(x), DeviceArray.from_numpy(y)):
        out = DeviceArray.empty((16384,), dt)
        ts = []
        for _ in range(4):
            device_sync()
            t = time.perf_counter()
            for _ in range(20):
                ops.reduce("amax", a, [1], out=out)
            device_sync()
            ts.append(time.perf_counter() - t)
        best.append(min(ts))
    assert best[1] < 10 * best[0]
