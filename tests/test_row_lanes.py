"""Fused rows of narrow types and of many elements: how many lanes share a row,
that every such row compiles, and its values.

A lane of the copied forms holds at most 128 elements of an integer operand
(uint8 rows of 65536 into bool have 512 at 128 lanes, past what the exact row
sums allow), and of rows over 512 vectors 288 registers of all operands
(integers counted with their converted values, bfloat16 packed).
"""
from __future__ import annotations

import re

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300._ffi import last_kernels
from xtensor_gb300.device import DeviceArray

from util import bf16_bits_to_f32, f32_to_bf16_bits, rng


@pytest.fixture
def dry():
    xg.set_option("jit.dry_run", 1)
    yield
    xg.set_option("jit.dry_run", -1)


def plan(dt, cols, operands=1):
    a = [DeviceArray((40000, cols), dt, (k + 1) << 36) for k in range(operands)]
    e = a[0]
    for x in a[1:]:
        e = e + x
    xg.assign(DeviceArray((40000, cols), "bool", 1 << 44), e > xg.rmean(e))
    name = last_kernels()[0]
    bulk = name.startswith("k_rowfused_tma")
    m = re.search(r", bool, (\d+), (\d+), (.*)>$", name)
    vec, nv, rest = int(m[1]), int(m[2]), m[3].split(", ")
    return bulk, int(rest[3] if bulk else rest[0]), vec * nv  # bulk copies, lanes, elements per lane


@pytest.mark.parametrize("cols", [4096, 8192, 16384, 32768, 65536])
def test_whole_vectors_of_bytes_compile(dry, cols):
    bulk, lanes, elems = plan("uint8", cols)
    assert elems <= (128 if bulk else 256)


@pytest.mark.parametrize("dt,cols,operands", [("uint8", 4095, 1), ("int16", 4095, 1), ("uint8", 16384, 3), ("int16", 32768, 1),
                                              ("float32", 16384, 3), ("float32", 8192, 1), ("bfloat16", 32768, 3), ("float64", 8192, 3)])
def test_lanes_hold_their_rows(dry, dt, cols, operands):
    bulk, lanes, elems = plan(dt, cols, operands)
    regs = {"uint8": 2, "int16": 2, "bfloat16": 0.5, "float32": 1, "float64": 2}[dt]
    assert not bulk or elems * operands * regs <= 288


@pytest.mark.gpu
@pytest.mark.parametrize("cols", [1001, 3001, 3073, 4095, 4096, 8192, 16384, 24576, 32768, 65536])
@pytest.mark.parametrize("dt", ["uint8", "int8", "int16", "bfloat16"])
def test_values(dt, cols):
    """x > mean(x) and x - max(x): exact, the means lie between two integers."""
    if cols > 4096 * (16 if dt in ("uint8", "int8") else 8):
        pytest.skip("longer than a fused row may be")
    g = rng(cols)
    x = g.integers(0, 100, (5, cols))
    mean = x.mean(1, keepdims=True)
    x[np.abs(mean[:, 0] - np.rint(mean[:, 0])) < 1e-3, 0] ^= 1  # (no mean at an integer)
    mean = x.mean(1, keepdims=True)
    assert (np.abs(mean - np.rint(mean)) > 1e-6).all()
    bits = f32_to_bf16_bits(x.astype(np.float32)) if dt == "bfloat16" else x.astype(dt)
    d = DeviceArray.from_numpy(bits, dt) if dt == "bfloat16" else DeviceArray.from_numpy(bits)
    o = DeviceArray.empty(x.shape, "bool")
    xg.assign(o, d > xg.rmean(d))
    np.testing.assert_array_equal(o.to_numpy().astype(bool), x > mean)
    o = DeviceArray.empty(x.shape, dt)
    if dt == "uint8":
        xg.assign(o, xg.ramax(d) - d)
        np.testing.assert_array_equal(o.to_numpy(), x.max(1, keepdims=True) - x)
    else:
        xg.assign(o, d - xg.ramax(d))
        got = o.to_numpy()
        got = bf16_bits_to_f32(got.view(np.uint16)) if dt == "bfloat16" else got
        np.testing.assert_array_equal(got, x - x.max(1, keepdims=True))
