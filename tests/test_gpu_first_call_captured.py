"""A stream that is being captured takes a call whose kind has not run before:
what the library keeps for its calls (scratch, the error word) exists from
xtg_init on, since a capture allows no such allocation.  A fresh process per
call, under torch's graph capture."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

ROOT = Path(__file__).resolve().parent.parent
SCRIPT = """
import sys
import torch
import xtensor_gb300 as xg
from xtensor_gb300 import ops
from xtensor_gb300.device import DeviceArray

def dev(t):
    return DeviceArray(tuple(t.shape), "float32", t.data_ptr(), base=t)

xg.init(0)
what = sys.argv[1]
x = torch.arange(8192 * 64, device="cuda", dtype=torch.float32).reshape(8192, 64) % 7
out = torch.zeros({"rows": (8192,), "whole": (), "fused": (8192, 64)}[what], device="cuda")
s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(g, stream=s):
    if what == "rows":
        ops.reduce("sum", dev(x), [1], out=dev(out), stream=s.cuda_stream)
    elif what == "whole":
        ops.reduce("sum", dev(x), out=dev(out), stream=s.cuda_stream)
    else:
        xg.assign(dev(out), dev(x) - xg.ramax(dev(x)), stream=s.cuda_stream)
for _ in range(2):
    out.fill_(-1)
    g.replay()
torch.cuda.synchronize()
want = {"rows": x.sum(1), "whole": x.sum(), "fused": x - x.amax(1, keepdim=True)}[what]
assert torch.equal(out, want)
"""


@pytest.mark.parametrize("what", ["rows", "whole", "fused"])
def test_first_call(what):
    r = subprocess.run([sys.executable, "-c", SCRIPT, what], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
