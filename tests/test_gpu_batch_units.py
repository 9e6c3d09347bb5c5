"""The streamed form of batched row reductions: instances at every phase of a
16-byte granule, instances inside one granule, rows of one element to several
units, leaves beside the streamed ones, strided results.

Tolerances: integers and maxima exact, float32 sums within 1e-6 of sum|x|
(those of the batch tests).
"""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300.batch import Batch
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (3, 1), (1, 3), (2, 2), (5, 3), (700, 1), (333, 2), (41, 5), (9, 16), (130, 31), (64, 64), (7, 127), (19, 129), (33, 300),
          (3, 1025), (2, 2500), (1, 4097)]


def carve(g, dt, draw):
    """(host, device) arrays of SHAPES, each at another phase of one buffer."""
    host, at, n = [], [], 0
    for k, (r, c) in enumerate(SHAPES):
        n = -(-n // 16) * 16 + k % 5
        host.append(draw((r, c)).astype(dt))
        at.append(n)
        n += r * c
    flat = np.full(n + 16, 99, dt)
    for h, a in zip(host, at):
        flat[a:a + h.size] = h.ravel()
    d = DeviceArray.from_numpy(flat)
    return host, [d[a:a + h.size].reshape(h.shape) for h, a in zip(host, at)]


@pytest.mark.parametrize("autotune", [False, True])
@pytest.mark.parametrize("dt", ["float32", "int32"])
def test_sums(dt, autotune, tmp_path, monkeypatch):
    monkeypatch.setenv("XTG_CACHE_DIR", str(tmp_path))
    g = rng(3)
    draw = (lambda s: g.standard_normal(s)) if dt == "float32" else (lambda s: g.integers(-99, 100, s))
    hA, dA = carve(g, dt, draw)
    hC, dC = carve(g, dt, draw)
    v = [draw(s[1]).astype(dt) for s in SHAPES]
    w = [draw((s[0], 1)).astype(dt) for s in SHAPES]
    dv, dw = [DeviceArray.from_numpy(x) for x in v], [DeviceArray.from_numpy(x) for x in w]
    outs = [DeviceArray.from_numpy(np.full(2 * s[0], 7, dt)) for s in SHAPES]
    b = Batch(dA[0] * dv[0] + dC[0] * dw[0], reduce="sum")
    for k in range(len(SHAPES)):
        b.add(dA[k] * dv[k] + dC[k] * dw[k], outs[k][::2])
    b.build(autotune=autotune)
    for _ in range(2):
        b.run()
    for k in range(len(SHAPES)):
        e = hA[k].astype(np.float64) * v[k] + hC[k].astype(np.float64) * w[k]
        got = outs[k].to_numpy()
        assert (got[1::2] == 7).all()
        tol = 0 if dt == "int32" else 1e-6 * (np.abs(hA[k] * v[k]) + np.abs(hC[k] * w[k])).sum(1)
        assert (np.abs(got[::2] - e.sum(1)) <= tol).all(), SHAPES[k]


@pytest.mark.parametrize("dt", ["float64", "uint8"])
def test_maxima_of_wide_and_narrow_types(dt):
    g = rng(4)
    draw = (lambda s: g.standard_normal(s)) if dt == "float64" else (lambda s: g.integers(0, 256, s))
    hA, dA = carve(g, dt, draw)
    outs = [DeviceArray.empty((s[0],), dt) for s in SHAPES]
    b = Batch(dA[0], reduce="amax")
    for d, o in zip(dA, outs):
        b.add(d, o)
    b.build(autotune=False)
    b.run()
    for h, o in zip(hA, outs):
        np.testing.assert_array_equal(o.to_numpy(), h.max(1))
