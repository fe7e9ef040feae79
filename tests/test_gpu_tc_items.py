"""The tensor-core contraction's work items.

* Items without a slice: a tile of one slice of functions cut into eight items
  leaves seven of them empty, so a CTA takes many in a row; results against the
  FP64 oracle, and the same to the last bit in every repetition.
* The same tiles in calls of different sizes, cut into different numbers of
  items: a slice's sums have a place of their own and are added in the order of
  the slices, so the results are equal to the last bit.  Grid spacing and origin
  are multiples of 1/8, so a slab's points are the whole grid's."""
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


@pytest.mark.parametrize("keys,per_tile", [(("rho",), 128), (KEYS, 32)])
@pytest.mark.parametrize("tiles", [1, 19, 147])  # fewer than 148: eight items each
def test_items_without_slices(torch_cuda, keys, per_tile, tiles):
    mol = S.make_molecule("c2", seed=4, natom=3, box=5.0, nocc=6)
    assert mol.nbasis <= 64
    pts = S.random_points(np.random.default_rng(tiles), mol, tiles * per_tile - 5, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    few = pts[:200]
    ref = O.eval_local(mol.flat(), mol.D, few, alpha=0.5, keys=KEYS)
    sc = term_scales(mol.flat(), mol.D, few, alpha=0.5)
    first = m.eval_local(pts, keys, ctc_abi.PREC_TC)
    for k in keys:
        assert np.isfinite(first[k]).all()
        assert_close(k, first[k][:200], ref[k], sc[k], 1e-8, atol=1e-15)
    for _ in range(50):
        again = m.eval_local(pts, keys, ctc_abi.PREC_TC)
        for k in keys:
            assert np.array_equal(again[k], first[k])
    assert m.sync_status() == 0


@pytest.mark.parametrize("keys", [("rho",), ("rho", "grad"), ("rho", "lap")])
def test_number_of_items_does_not_change_results(torch_cuda, keys):
    mol = S.make_molecule("c2", seed=9, natom=30, box=11.0, nocc=60)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    shape, h = (48, 32, 40), 0.375  # 1 920 tiles of 32 points or 480 of 128
    origin = np.round(8.0 * mol.coords.mean(0)) / 8.0 - 8.0
    axes = h * np.eye(3)
    whole = m.eval_cubic(origin, axes, shape, keys=keys, precision=ctc_abi.PREC_TC)
    for x0, nx in ((0, 4), (16, 4), (20, 12)):
        part = m.eval_cubic(origin + x0 * axes[0], axes, (nx,) + shape[1:], keys=keys, precision=ctc_abi.PREC_TC)
        for k in keys:
            w = whole[k].reshape(shape[0], -1)[x0:x0 + nx].ravel()
            assert np.array_equal(part[k], w), k


@pytest.mark.parametrize("keys,per_tile", [(("rho",), 128), (KEYS, 32)])
@pytest.mark.parametrize("near,far", [(1, 140), (12, 90), (40, 40)])
def test_tiles_of_very_different_sizes(torch_cuda, keys, per_tile, near, far):
    """Tiles near the molecule (several slices, cut into up to eight items) among
    tiles that keep few functions or none, whose further items are empty."""
    mol = S.make_molecule("c2", seed=6, natom=30, box=11.0, nocc=60)
    rng = np.random.default_rng(near)
    pts = np.concatenate([S.random_points(rng, mol, near * per_tile, pad=0.5),
                          mol.coords.mean(0) + np.array([22.0, 0.0, 0.0]) + rng.uniform(-9, 9, (far * per_tile, 3))])
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    few = np.r_[0:min(100, near * per_tile), len(pts) - 50:len(pts)]
    ref = O.eval_local(mol.flat(), mol.D, pts[few], alpha=0.5, keys=KEYS)
    sc = term_scales(mol.flat(), mol.D, pts[few], alpha=0.5)
    first = m.eval_local(pts, keys, ctc_abi.PREC_TC)
    for k in keys:
        assert np.isfinite(first[k]).all()
        assert_close(k, first[k][few], ref[k], sc[k], 1e-8, atol=1e-15)
    for _ in range(50):
        again = m.eval_local(pts, keys, ctc_abi.PREC_TC)
        for k in keys:
            assert np.array_equal(again[k], first[k])
    assert m.sync_status() == 0
