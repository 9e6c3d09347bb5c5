"""Registers of the row reductions whose speed is the number of resident blocks:
64 of them for four blocks of 256 threads per SM, 85 for three."""
from __future__ import annotations

import re
import subprocess
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

from xtensor_gb300.build import cuda_home

CSRC = Path(__file__).resolve().parent.parent / "xtensor_gb300" / "csrc"

# leaf type, accumulator, result, vector, reduced dims, lanes, registers at most
FORMS = [("double", "AccPlain<double, 0>", "double", 2, 1, 256, 64),
         ("double", "AccSel<double, 1>", "double", 2, 1, 256, 64),
         ("double", "AccSel<double, 1>", "double", 2, 2, 32, 64),
         ("float", "AccSel<float, 1>", "float", 4, 2, 32, 64),
         ("xtg::bf16", "AccMom<float, 1>", "double", 8, 2, 16, 85)]


def registers(args):
    k, (leaf, acc, out, vec, rr, lanes, _), tmp = args
    src = tmp / f"form{k}.cu"
    src.write_text(f'#include "xtg_device.cuh"\n'
                   f"template __global__ void xtg::k_reduce_row<xtg::L<0, {leaf}>, xtg::LeafSet<xtg::LeafSpec<{leaf}, 0>>, "
                   f"xtg::{acc}, {out}, 0, {vec}, 1, {rr}, {lanes}, false, 4>(const xtg::RedParams);\n")
    cmd = [str(cuda_home() / "bin" / "nvcc"), "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false",
           "-Xptxas", "-v", "-I", str(CSRC), "-I", str(CSRC.parent.parent / "include"), "-c", str(src),
           "-o", str(tmp / f"form{k}.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return max(int(n) for n in re.findall(r"Used (\d+) registers", r.stderr))


def test_registers(tmp_path):
    with ThreadPoolExecutor() as pool:
        used = list(pool.map(registers, [(k, f, tmp_path) for k, f in enumerate(FORMS)]))
    assert all(n <= f[-1] for n, f in zip(used, FORMS)), list(zip(FORMS, used))
