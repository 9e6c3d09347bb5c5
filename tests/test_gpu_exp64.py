"""exp of float64: within 0.51 ulp of the exact value (0.503 by its derivation)
over all magnitudes, subnormal results included; the ends and the specials as
the library's."""
from __future__ import annotations

import numpy as np
import pytest

import xtensor_gb300 as xg
from xtensor_gb300.device import DeviceArray

from util import rng

pytestmark = pytest.mark.gpu


def run(x):
    d = DeviceArray.from_numpy(x)
    out = DeviceArray.from_numpy(np.zeros_like(x))
    xg.assign(out, xg.exp(d))
    return out.to_numpy()


@pytest.mark.parametrize("kind", ["wide", "near", "small", "steps", "subnormal"])
def test_error(kind):
    g = rng(5)
    n = 20011
    step = np.log(2.0) / 64
    x = {
        "wide": g.uniform(-708.3, 709.7, n),
        "near": g.standard_normal(n),
        "small": g.choice([-1.0, 1.0], n) * 2.0 ** g.uniform(-80, 0, n),
        "steps": np.nextafter(g.integers(-65000, 65000, n) * step, g.choice([-1e3, 0, 1e3], n)),
        "subnormal": g.uniform(-745.2, -708.3, n),
    }[kind]
    got = run(x)
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("no wider type to compare with")
    exact = np.exp(x.astype(np.longdouble))
    ulp = np.spacing(np.maximum(exact.astype(np.float64), 2.0**-1022))
    assert (np.abs(got - exact) <= 0.51 * ulp).all()


def test_ends():
    top, low = 709.782712893384, -745.1332191019411
    x = np.array([0.0, -0.0, 5e-324, -5e-324, top, np.nextafter(top, 1e3), low, -745.1332191019412, 1023.9, 1024.0, -1023.9,
                  -1e4, 1e300, -1e300, np.inf, -np.inf, np.nan])
    with np.errstate(all="ignore"):
        want = np.exp(x)
    np.testing.assert_array_equal(run(x), want)
