"""Batched row sums of many wide operands: whatever form the build chooses (and
the tuner tries), its buffers fit a block's shared memory.  The data are small
integers, so every sum is exact in any order."""
from __future__ import annotations

from functools import reduce as fold

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300.batch import Batch, fill_random
from xtensor_gb300.device import DeviceArray

pytestmark = pytest.mark.gpu

# (rows, columns) of the instances: a few rows; enough for the largest units
SMALL = [(5, 70), (33, 129), (1, 1000)]
LARGE = [(1024, 601 + i) for i in range(16)]


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("dt,operands,shapes", [("float64", 3, SMALL), ("float64", 3, LARGE), ("float32", 8, SMALL),
                                                ("float32", 8, LARGE), ("float32", 5, LARGE)])
def test_sums(dt, operands, shapes, autotune, tmp_path, monkeypatch):
    monkeypatch.setenv("XTG_CACHE_DIR", str(tmp_path))
    check(dt, operands, shapes, autotune)


def test_large_tiles_asked_for():
    xg.set_option("batch.tile_elems", 8192)
    try:
        check("float64", 2, LARGE, False)
    finally:
        xg.set_option("batch.tile_elems", -1)


def test_the_streamed_form_asked_for_where_nothing_streams():
    xg.set_option("batch.group_lanes", 0)
    try:
        x = fill_random(DeviceArray.empty((40, 30), "float32"), "integers", -4, 4, 1)
        y = DeviceArray.empty((40, 30), "float32")
        b = Batch(x + x)
        b.add(x + x, y)
        b.build(autotune=False)
        b.run()
        np.testing.assert_array_equal(y.to_numpy(), 2 * x.to_numpy())
    finally:
        xg.set_option("batch.group_lanes", -1)


def check(dt, operands, shapes, autotune):
    arrays = [[fill_random(DeviceArray.empty(s, dt), "integers", -4, 4, 100 * i + k) for k in range(operands)]
              for i, s in enumerate(shapes)]
    outs = [DeviceArray.empty((s[0],), dt) for s in shapes]

    def expr(a):
        return fold(lambda x, y: x + y, a[2:], a[0] * a[1])

    b = Batch(expr(arrays[0]), reduce="sum")
    for a, o in zip(arrays, outs):
        b.add(expr(a), o)
    b.build(autotune=autotune)
    b.run()
    for a, o in zip(arrays, outs):
        np.testing.assert_array_equal(o.to_numpy(), ops.reduce("sum", expr(a), [1]).to_numpy())
