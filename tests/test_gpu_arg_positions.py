"""Arg-reductions past 2^32 elements: positions need more than 32 bits, and
among equal values the first one wins on either side of 2^32."""
from __future__ import annotations

import pytest

import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

pytestmark = pytest.mark.gpu

N = 2**32 + 5


def put(d, at, v):
    for i in at:
        xg.assign(d[i:i + 1], xg.scalar(v, d_type(d)))


def d_type(d):
    return "int8" if d.itemsize == 1 else "float64"


@pytest.mark.parametrize("dt", ["int8", "float64"])
@pytest.mark.parametrize("at", [[2**32 + 1], [2**32 + 4], [2**32 - 1, 2**32 + 1], [9, 2**32 + 3], [2**32, 2**32 + 2]])
def test_whole_array(dt, at):
    d = DeviceArray.empty((N,), dt)
    xg.assign(d, xg.scalar(1, dt))
    put(d, at, 3)
    assert int(ops.argreduce("argmax", d).to_numpy()) == at[0]
    put(d, at, -3)
    assert int(ops.argreduce("argmin", d).to_numpy()) == at[0]


def test_rows():
    d = DeviceArray.empty((2, N), "int8")
    xg.assign(d, xg.scalar(0, "int8"))
    put(d.reshape((2 * N,)), [N - 2, N + 7, 2 * N - 3], 5)
    assert ops.argreduce("argmax", d, 1).to_numpy().tolist() == [N - 2, 7]
    put(d.reshape((2 * N,)), [N + 7], 0)
    assert ops.argreduce("argmax", d, 1).to_numpy().tolist() == [N - 2, N - 3]
