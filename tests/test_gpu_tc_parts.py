"""The tensor-core contraction's work items: few tiles (a tile's slices dealt out
to up to eight items), many tiles, fewer slices than items, and padding in the
last slice, against the FP64 oracle; and the same points in calls of different
sizes, whose tiles are cut into different numbers of items, bit for bit where
the tiles are the same."""
import numpy as np
import pytest

import ctc_abi
from helpers import assert_close, term_scales
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu
KEYS = ("rho", "grad", "hess", "lap", "tau_pd")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("natom", [2, 5, 12, 40])  # one slice of functions up to about ten
@pytest.mark.parametrize("n", [1, 31, 200, 3000])
def test_items_per_tile(torch_cuda, natom, n):
    mol = S.make_molecule("c2", seed=natom, natom=natom, box=3.0 * natom ** (1 / 3) + 1.5, nocc=2 * natom)
    pts = S.random_points(np.random.default_rng(n), mol, n, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    few = pts[:200]
    ref = O.eval_local(mol.flat(), mol.D, few, alpha=0.5, keys=KEYS)
    sc = term_scales(mol.flat(), mol.D, few, alpha=0.5)
    for keys in (("rho",), ("rho", "grad"), KEYS):
        got = m.eval_local(pts, keys, ctc_abi.PREC_TC)
        for k in keys:
            assert np.isfinite(got[k]).all()
            assert_close(k, got[k][:200], ref[k], sc[k], 1e-8, atol=1e-15)
    assert m.sync_status() == 0


def test_items_do_not_change_results(torch_cuda):
    """The same grid in slabs: tiles of two planes, the same blocks in every call."""
    mol = S.make_molecule("c2", seed=9, natom=30, box=11.0, nocc=60)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    origin, axes = S.cube_grid(mol, 0.35, (24, 28, 28))
    whole = m.eval_cubic(origin, axes, (24, 28, 28), keys=("rho", "lap"), precision=ctc_abi.PREC_TC)
    for x0, nx in ((0, 2), (4, 8)):
        part = m.eval_cubic(origin + x0 * axes[0], axes, (nx, 28, 28), keys=("rho", "lap"), precision=ctc_abi.PREC_TC)
        for k in part:
            w = whole[k].reshape(24, -1)[x0:x0 + nx].ravel()
            # the slab's origin is rounded, so its points are the grid's to 1e-15
            np.testing.assert_allclose(part[k], w, rtol=0, atol=1e-9 * np.abs(w).max())
    again = m.eval_cubic(origin, axes, (24, 28, 28), keys=("rho", "lap"), precision=ctc_abi.PREC_TC)
    for k in again:
        assert np.array_equal(again[k], whole[k])
