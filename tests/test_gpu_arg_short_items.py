"""Arg-reductions by blocks whose last work item has fewer vectors than the
block has threads: a thread without elements holds no value."""
from __future__ import annotations

import numpy as np
import pytest

from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

# 2048 work items of 2100 vectors of two float64, the last of `last` vectors
CHUNK = 2100


@pytest.mark.parametrize("last", [1, 31, 100, 255])
@pytest.mark.parametrize("dt", ["float64", "float32", "int64"])
def test_last_item(dt, last):
    vec = 4 if dt == "float32" else 2
    n = (2047 * CHUNK + last) * vec + 1
    x = rng(last).integers(-1000, 1001, n).astype(dt)
    d = DeviceArray.from_numpy(x)
    for op in ("argmax", "argmin"):
        assert int(ops.argreduce(op, d).to_numpy()) == int(getattr(np, op)(x)), op
    x[-1], x[-vec - 1] = 2000, -2000  # in the last item
    d = DeviceArray.from_numpy(x)
    for op in ("argmax", "argmin"):
        assert int(ops.argreduce(op, d).to_numpy()) == int(getattr(np, op)(x)), op
