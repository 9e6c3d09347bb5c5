"""K13 and the one-pass moments at any length and alignment: bit for bit what
K3 gives (K13 folds its vectors in K3's order, whatever their width), and each
moment what its own reduction gives."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300._ffi import check, last_kernels
from xtensor_gb300.device import DeviceArray

from util import f32_to_bf16_bits, rng

pytestmark = pytest.mark.gpu


def data(n, dt):
    g = rng(n)
    x = (g.lognormal(0.0, 2.0, n) * np.where(g.random(n) < 0.5, -1.0, 1.0) + 1.0).astype(np.float32)
    return DeviceArray.from_numpy(f32_to_bf16_bits(x) if dt == "bfloat16" else x, dt)


@pytest.mark.parametrize("dt", ["float32", "bfloat16"])
@pytest.mark.parametrize("n", [1 << 25, (1 << 25) + 1, (1 << 25) + 8 * 4097 + 6, 3 * (1 << 24) - 3])
def test_stream_equals_row_kernel(dt, n):
    d = data(n + 7, dt)
    for off in (0, 1, 4, 7):
        v = d[off:off + n]
        for op in ("sum", "variance", "norm_l2"):
            a = ops.reduce(op, v).to_numpy()
            ks = last_kernels()
            assert ks[0].startswith("k_reduce_stream<"), ks
            xg.set_option("reduce.stream", 0)
            try:
                b = ops.reduce(op, v).to_numpy()
            finally:
                xg.set_option("reduce.stream", -1)
            assert a.tobytes() == b.tobytes(), (op, off)
    check(xg.lib().xtg_check_device_errors())


@pytest.mark.parametrize("chunk", [None, 64])
@pytest.mark.parametrize("dt", ["float32", "bfloat16"])
@pytest.mark.parametrize("n", [1, 5, 1000, 4099, 100003, 262145, 1 << 20, (1 << 22) + 3, (1 << 24) + 5])
def test_moments_equal_separate_reductions(dt, n, chunk):
    d = data(n + 3, dt)
    if chunk is not None:
        xg.set_option("reduce.cta_chunk", chunk)
    try:
        for off in (0, 3):
            v = d[off:off + n]
            got = ops.reduce_moments(v, ddof=1 if n > 1 else 0)
            assert len(last_kernels()) <= 2
            for nm in ops.MOMENTS:
                want = ops.reduce(nm, v, ddof=1 if n > 1 and nm == "variance" else 0).to_numpy()
                assert got[nm].to_numpy().tobytes() == want.tobytes(), (nm, off)
    finally:
        xg.set_option("reduce.cta_chunk", -1)
    check(xg.lib().xtg_check_device_errors())
