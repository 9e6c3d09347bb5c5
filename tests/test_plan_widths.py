"""Vector widths and row groups that the planner takes where wider ones lose."""
from __future__ import annotations

import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray


@pytest.fixture(autouse=True)
def dry():
    xg.set_option("jit.dry_run", 1)
    yield
    xg.set_option("jit.dry_run", -1)


@pytest.mark.parametrize("dt,op,vec", [("int8", "sum", 8), ("int8", "amax", 4), ("int16", "amax", 4), ("bfloat16", "amax", 4),
                                       ("int16", "sum", 8), ("float64", "amax", 2), ("int32", "sum", 4)])
@pytest.mark.parametrize("n", [1 << 26, (1 << 26) - 3])
def test_whole_arrays(dt, op, vec, n):
    x = DeviceArray((n,), dt, 1 << 36)
    shape, rt = ops.reduce_shape(op, x)
    ops.reduce(op, x, out=DeviceArray(shape, rt, 1 << 40))
    assert f", {vec}, 1, 1, 256, " in last_kernels()[0]


@pytest.mark.parametrize("dt,inner,groups", [("float32", 2, False), ("float32", 3, True), ("bfloat16", 2, True)])
def test_groups_of_rows(dt, inner, groups):
    x = DeviceArray((1000, 88, inner + 3), dt, 1 << 36)[:, :, :inner]
    xg.assign(DeviceArray((1000, 88, inner), dt, 1 << 40), x)
    assert last_kernels()[0].endswith(", true>") == groups
