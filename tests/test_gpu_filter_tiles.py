"""Filters at the edges of their tiles (4096 positions, 512 per warp, 4096
tiles per step of the scan), over every alignment and selectivity; float32
comparisons with float64 scalars.  Everything is exact."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 511, 512, 513, 4095, 4096, 4097, 70001, 4096 * 4096 + 4097])
@pytest.mark.parametrize("dt", ["float32", "float64", "uint8"])
def test_reads_and_writes(dt, n):
    g = rng(n)
    x = (g.integers(0, 200, n + 1) if dt == "uint8" else g.integers(-100, 100, n + 1) * 0.5).astype(dt)
    d = DeviceArray.from_numpy(x)
    for off in ((0, 1) if n < 100000 else (0,)):
        v, h = d[off:off + n], x[off:off + n]
        for cut in (1000.0, 45.0, 0.0, -1000.0):
            keep = h > cut
            c = v > cut if dt != "uint8" else xg.cast(v, "float64") > cut
            assert ops.filter_count(c) == int(keep.sum())
            np.testing.assert_array_equal(ops.filter(v, c).to_numpy(), h[keep])
            np.testing.assert_array_equal(ops.filter(v + v, c).to_numpy(), (h + h if dt != "uint8" else h.astype(np.int32) * 2)[keep])  # uint8 promotes to int
            z = DeviceArray.from_numpy(x)
            ops.filter_assign(z[off:off + n], c, xg.scalar(3, dt))
            want = x.copy()
            want[off:off + n][keep] = 3
            np.testing.assert_array_equal(z.to_numpy(), want)
            src = g.integers(0, 50, int(keep.sum())).astype(dt)
            if 1 < src.size < 100000:
                ops.filter_assign(z[off:off + n], c, DeviceArray.from_numpy(src), "+=")
                want[off:off + n][keep] += src
                np.testing.assert_array_equal(z.to_numpy(), want)


def test_views_other_leaves_and_lengths():
    g = rng(2)
    x, y = g.standard_normal((2, 67, 301)).astype(np.float32)
    dx, dy = DeviceArray.from_numpy(x), DeviceArray.from_numpy(y)
    keep = x[3:, ::2] > 0.25
    got = ops.filter(dy[3:, ::2], dx[3:, ::2] > 0.25).to_numpy()
    np.testing.assert_array_equal(got, y[3:, ::2][keep])
    got = ops.filter(dy.transpose() + 1.0, dx.transpose() > 0.25).to_numpy()
    np.testing.assert_array_equal(got, (y.T.astype(np.float64) + 1.0).astype(got.dtype)[x.T > 0.25])
    # another length is refused, and the destination stays as it was
    out = DeviceArray.from_numpy(np.full(int((x > 0.25).sum()) + 1, 7, np.float32))
    with pytest.raises(xg.XtgError) as ei:
        ops.filter(dx, dx > 0.25, out=out)
    assert ei.value.status == 5
    assert (out.to_numpy() == 7).all()


def test_float32_against_float64_scalars():
    """Every comparison with a double scalar, either way around, is the
    comparison in double."""
    ds = [0.1, 0.0, -0.0, 1.0, 1 / 3, -1 / 3, 1e-46, -1e-46, 1.4e-45, 3.4028235e38, 3.41e38, -3.41e38, 1e300, np.inf, -np.inf, np.nan]
    near = np.concatenate([[np.nextafter(np.float32(d), np.float32(s)) for s in (-np.inf, np.inf)] + [np.float32(d)]
                           for d in ds[:10]] + [np.float32([np.inf, -np.inf, np.nan, 3.4028235e38, -3.4028235e38])]).astype(np.float32)
    x = np.concatenate([near, rng(1).standard_normal(5000).astype(np.float32)])
    dx, w = DeviceArray.from_numpy(x), x.astype(np.float64)
    from xtensor_gb300.expr import E, OP, as_expr
    with np.errstate(over="ignore", invalid="ignore"):
        for d in ds:
            for op, f in (("LT", np.less), ("LE", np.less_equal), ("GT", np.greater), ("GE", np.greater_equal),
                          ("EQ", np.equal), ("NE", np.not_equal)):
                s = xg.scalar(float(d))
                for e, want in ((E(OP[op], (as_expr(dx), s)), f(w, d)), (E(OP[op], (s, as_expr(dx))), f(d, w))):
                    np.testing.assert_array_equal(ops.filter(dx, e).to_numpy(), x[want], err_msg=f"{op} {d}")
