"""The kernels that place a unit's first and last elements beside its bulk copy
by plain stores of their lanes: other lanes read them, and neither a warp vote
nor the wait for the copy orders those stores.  A warp or block barrier has to
lie between the stores and the first read of the unit, in each kernel."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parent.parent / "xtensor_gb300" / "csrc" / "xtg_device.cuh").read_text()
BARRIER = re.compile(r"^\s*(?:if \([^)]*\) )?__sync(?:warp|threads)\(\);", re.M)


def body(kernel):
    at = re.search(r"\b%s\(const \w+ p\) \{" % kernel, SRC).end()
    return SRC[at:SRC.index("\n}\n", at)]


@pytest.mark.parametrize("kernel,store,read", [
    ("k_rowfused_tma", "E::store(edge", "LoadRowSmem<LS>"),
    ("k_reduce_unit", "::E::run(src", "UnitLoads<LS>"),
    ("k_batch_rowunits", "BU::put_edges(ev", "mbar_expect_tx(&full"),  # handed on by the producer's arrival
])
def test_a_barrier_follows_the_ends(kernel, store, read):
    text = re.sub(r"//[^\n]*", "", body(kernel))
    stored = text.index(store)
    assert BARRIER.search(text[stored:text.index(read, stored)]), kernel
