"""Comparisons of float64 as integers: numpy's results for every pair of
specials and neighbours, as arrays and against scalars."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300.device import DeviceArray

pytestmark = pytest.mark.gpu

S = np.array([0.0, -0.0, 5e-324, -5e-324, 1.0, -1.0, np.nextafter(1, 2), -np.nextafter(1, 2), 1e308, -1e308, np.inf, -np.inf,
              np.nan, -np.nan, 2.0**-1022, np.nextafter(2.0**-1022, 0)])
S = np.concatenate([S, np.array([0x7FF0000000000001, 0xFFF0000000000001, 0xFFFFFFFFFFFFFFFF], np.uint64).view(np.float64)])
OPS = ["less", "less_equal", "greater", "greater_equal", "equal", "not_equal"]


def ev(e, shape):
    out = DeviceArray.from_numpy(np.zeros(shape, bool))
    xg.assign(out, e)
    return out.to_numpy()


def cmp(name, a, b):
    return {"less": lambda: a < b, "less_equal": lambda: a <= b, "greater": lambda: a > b, "greater_equal": lambda: a >= b,
            "equal": lambda: xg.equal(a, b), "not_equal": lambda: xg.not_equal(a, b)}[name]()


@pytest.mark.parametrize("name", OPS)
def test_pairs(name):
    a, b = np.repeat(S, S.size), np.tile(S, S.size)
    with np.errstate(invalid="ignore"):
        want = getattr(np, name)(a, b)
        np.testing.assert_array_equal(ev(cmp(name, DeviceArray.from_numpy(a), DeviceArray.from_numpy(b)), a.shape), want)
        for v in S:
            got = ev(cmp(name, DeviceArray.from_numpy(S), xg.scalar(float(v), "float64")), S.shape)
            np.testing.assert_array_equal(got, getattr(np, name)(S, v))
