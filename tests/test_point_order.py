"""Rules for ordering explicit points (chemtoolscuda_b200/csrc/ctc_chunk.h,
compiled here with the host compiler).  The Morton keys' cells follow the box: on
long molecules tiles of 32 consecutive points are as compact as with 30-bit
keys, also when all points lie near one end."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "ctc_chunk.h"
extern "C" int axis_bits(double ext) { return ctc::morton_axis_bits(ext); }
extern "C" int sorted(long long n, int mpad, double ext) { return ctc::sort_points(n, mpad, ext); }
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "r.cpp").write_text(SRC)
    so = str(d / "r.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", str(d / "r.cpp"), "-o", so,
                    "-I" + os.path.join(ROOT, "chemtoolscuda_b200", "csrc")], check=True)
    L = C.CDLL(so)
    L.axis_bits.argtypes = [C.c_double]
    L.sorted.argtypes = [C.c_longlong, C.c_int, C.c_double]
    return L


def _mean_tile_radius(pts, lo, ext, bits):
    q = np.clip((pts - lo) * (2 ** bits / ext), 0, 2 ** bits - 1).astype(np.uint64)
    key = np.zeros(len(pts), np.uint64)
    for b in range(bits):
        for d in range(3):
            key |= ((q[:, d] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + d)
    p = pts[np.argsort(key, kind="stable")][:len(pts) // 32 * 32].reshape(-1, 32, 3)
    c = p.mean(axis=1, keepdims=True)
    return np.sqrt(((p - c) ** 2).sum(-1).max(1)).mean()


@pytest.mark.parametrize("length", [20.0, 150.0, 480.0, 1500.0, 6000.0])
@pytest.mark.parametrize("end", [False, True])
def test_tiles_of_long_molecules_stay_compact(rules, length, end):
    rng = np.random.default_rng(int(length))
    hi = np.array([length, 6.0, 6.0])
    pts = rng.uniform(-3.0, np.minimum(hi, 100.0) if end else hi, (200_000, 3))
    lo, ext = np.full(3, -12.0), length + 24.0
    fine = _mean_tile_radius(pts, lo, ext, 10)
    assert _mean_tile_radius(pts, lo, ext, rules.axis_bits(ext)) <= 1.15 * fine


def test_cells(rules):
    for ext in np.exp(np.linspace(np.log(24.0), np.log(1e5), 400)):
        bits = rules.axis_bits(ext)
        assert bits in (8, 10)  # 24 or 30 bits in all: spread10 and 32-bit keys hold both
        assert ext / 2 ** bits <= max(2.0, ext / 1024)
    assert rules.axis_bits(float("nan")) == 10


def test_small_calls_of_spread_out_molecules_are_sorted(rules):
    """Unsorted only where a tile keeps most functions in any order: few points, few
    functions, and a molecule of at most 40 bohr (64 with its padding)."""
    assert not rules.sorted(2048, 256, 64.0) and not rules.sorted(1, 128, 24.0)
    assert rules.sorted(2049, 128, 24.0) and rules.sorted(1, 384, 24.0)
    assert rules.sorted(1, 128, 64.1) and rules.sorted(2048, 256, 1000.0) and rules.sorted(1, 128, float("nan"))
