"""Full reductions whose length (or address) vectors do not divide keep the
accuracy of element-by-element sums: means and norms of odd lengths within
1e-12 (double-float: 2^-45 and the roundings of its combination), small,
streamed and misaligned."""
from __future__ import annotations

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1001, 100_003, 1_000_001, 3_000_001, (1 << 23) + 1])
def test_odd_lengths(n):
    x = rng(n).lognormal(0.0, 2.0, n + 1).astype(np.float32)
    d = DeviceArray.from_numpy(x)
    for v, h in ((d[:n], x[:n]), (d[1:], x[1:]), (d[1:n], x[1:n])):
        w = h.astype(np.longdouble)
        if h.size % 2:
            assert abs(float(ops.reduce("norm_l2", v, None).to_numpy()) - np.sqrt((w * w).sum())) <= 1e-12 * np.sqrt((w * w).sum())
        assert abs(float(ops.reduce("mean", v, None).to_numpy()) - w.mean()) <= 1e-12 * w.mean()
