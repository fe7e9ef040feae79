"""Chunks of the tile pipeline (chemtoolscuda_b200/csrc/ctc_chunk.h, compiled
here with the host compiler): within the budget, in whole rounds of one tile per
SM where that drops little of a chunk; and no question for the free device memory in a call whose block the molecule
holds already -- the second call of any size among them."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "ctc_chunk.h"
extern "C" {
long long tiles(unsigned long long budget, unsigned long long tile, long long ntiles, int sms) {
  return ctc::chunk_tiles(budget, tile, ntiles, sms);
}
int ask(unsigned long long block, unsigned long long held) { return ctc::ask_free_memory(block, held); }
unsigned long long most() { return ctc::kMostAo; }
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("chunk")
    (d / "plan.cpp").write_text(SRC)
    so = str(d / "plan.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", str(d / "plan.cpp"), "-o", so,
                    "-I" + os.path.join(ROOT, "chemtoolscuda_b200", "csrc")], check=True)
    L = C.CDLL(so)
    L.tiles.restype = C.c_longlong
    L.tiles.argtypes = [C.c_ulonglong, C.c_ulonglong, C.c_longlong, C.c_int]
    L.ask.argtypes = [C.c_ulonglong, C.c_ulonglong]
    L.most.restype = C.c_ulonglong
    return L


def test_chunks_fill_the_budget_in_whole_rounds_where_that_costs_little(plan):
    rng = np.random.default_rng(0)
    whole = 0
    for _ in range(5000):
        tile = int(np.exp(rng.uniform(np.log(1e4), np.log(3e8))))
        ntiles = int(np.exp(rng.uniform(0, np.log(1e6))))
        budget = int(np.exp(rng.uniform(np.log(1e6), np.log(2e10))))
        c = plan.tiles(budget, tile, ntiles, 148)
        assert 1 <= c <= ntiles
        if c < ntiles:
            most = max(148, budget // tile)
            assert 0.95 * most <= c <= most
            whole += c % 148 == 0
    assert whole > 500
    assert plan.tiles(12 << 30, 8 * 10 * 32 * 7040, 6250, 148) == (12 << 30) // (8 * 10 * 32 * 7040)  # 714


def test_second_call_does_not_ask(plan):
    """2 691 functions (2 816 padded), 32-point tiles, ten quantities: 1 776 of the
    1 787 tiles that 12 GiB hold; and blocks of any other shape."""
    most = plan.most()
    tile = 8 * 10 * 32 * 2816
    assert plan.tiles(most, tile, 10 ** 6, 148) == 1776
    rng = np.random.default_rng(1)
    shapes = [(tile, 10 ** 6)] + [(8 * int(nq) * int(tp) * 64 * int(k), int(nt)) for nq, tp, k, nt in zip(
        rng.choice([1, 2, 4, 10, 11], 3000), rng.choice([32, 64, 128], 3000), rng.integers(1, 260, 3000),
        np.exp(rng.uniform(0, np.log(1e6), 3000)))]
    for t, n in shapes:
        block = t * plan.tiles(most, t, n, 148)
        held = max(block, 1 << 20)  # what the first call left
        assert not plan.ask(block, held)
        assert plan.ask(block, 0) == (block > 64 << 20)
