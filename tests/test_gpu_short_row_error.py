"""Many short rows of float32 and bfloat16: their sums of squares and deviations
carry a TwoSum per element, so norms and sums are as exact as double-float
arithmetic: 32 elements at 2^-46 each, against the terms' size.  A variance's
deviations from the row's first element are float32 (2^-24 each, twice in a
square, and once more through their sum), whatever the sums."""
from __future__ import annotations

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

from util import bf16_bits_to_f32, f32_to_bf16_bits, rng

pytestmark = pytest.mark.gpu

BOUND = 32 * 2.0**-46


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("dt", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,cols", [(1024, 4), (5000, 8), (4099, 16), (4099, 24), (1500, 28), (4099, 30), (5000, 31)])
def test_rows(rows, cols, dt, fused):
    x = rng(cols).standard_normal((rows, cols)).astype(np.float32)
    if dt == "bfloat16":
        d = DeviceArray.from_numpy(f32_to_bf16_bits(x), dt)
        x = bf16_bits_to_f32(f32_to_bf16_bits(x))
    else:
        d = DeviceArray.from_numpy(x)
    L = x.astype(np.longdouble)
    dev = L - L[:, :1]
    for op, want, size in [("variance", np.square(L - L.mean(1, keepdims=True)).mean(1), np.square(dev).mean(1)),
                           ("norm_sq", np.square(L).sum(1), np.square(L).sum(1)),
                           ("norm_l1", np.abs(L).sum(1), np.abs(L).sum(1)),
                           ("mean", L.mean(1), np.abs(L).mean(1))]:
        if fused:
            got = ops.assign_reduce(DeviceArray.empty((rows, cols), dt), d, op, axes=[1]).to_numpy()
        else:
            got = ops.reduce(op, d, [1]).to_numpy()
        bound = 4 * 2.0**-24 if op == "variance" else BOUND if got.dtype == np.float64 else 2.0**-23
        assert (np.abs(got - want) <= bound * size).all(), (op, float((np.abs(got - want) / size).max()))
