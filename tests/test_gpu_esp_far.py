"""The ESP's far-field polynomials and the split of pairs into far and near.

A molecule with every class of pairs up to g-g, points from inside the molecule
to 200 bohr away (every pair near, every pair far, and blocks with both), point
counts around the 128- and 256-point blocks and the two-points-per-thread form,
against the FP64 oracle.  Tolerance: 1e-10 of the sum of absolute terms (the
nuclear part plus the electronic part), the ESP's tolerance elsewhere."""
import numpy as np
import pytest

import ctc_abi
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _molecule(lmax):
    rng = np.random.default_rng(31 + lmax)
    coords = np.array([[0.0, 0.0, 0.0], [2.2, 0.4, -0.3], [-0.9, 1.9, 1.2]])
    kinds = [am for am in (0, 1, 2, -2, 3, -3, 4, -4) if abs(am) <= lmax]
    shells = []
    for i, am in enumerate(kinds + [0, 1][:lmax + 1]):
        e = np.exp(rng.uniform(np.log(0.12), np.log(60.0), size=2))
        shells.append(S.Shell(center=coords[i % 3], atom=i % 3, angmoms=[am], exponents=e,
                              coeffs=rng.standard_normal((1, 2))))
    M = sum(S.nfunc(a) for s in shells for a in s.angmoms)
    z = np.array([8.0, 6.0, 1.0])
    return S.SyntheticMolecule(coords=coords, numbers=z.astype(np.int32), charges=z, shells=shells,
                               D=S.make_density_matrix(rng, M, max(1, M // 3)))


def _points(mol, n, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((n, 3))
    r = np.exp(rng.uniform(np.log(0.3), np.log(200.0), size=n))
    return mol.coords[rng.integers(0, 3, n)] + r[:, None] * v / np.linalg.norm(v, axis=1, keepdims=True)


def _check(mol, pts, got):
    ref = O.eval_esp(mol.flat(), mol.D, mol.coords, mol.charges, pts)
    nuc = (mol.charges / np.linalg.norm(pts[:, None] - mol.coords[None], axis=-1)).sum(1)
    assert (np.abs(got - ref) <= 1e-10 * (nuc + np.abs(nuc - ref)) + 1e-15).all(), np.abs(got - ref).max()


@pytest.mark.parametrize("n", [1, 127, 129, 300])
@pytest.mark.parametrize("lmax", [0, 1, 2, 3, 4])
def test_classes_and_block_sizes(torch_cuda, lmax, n):
    mol = _molecule(lmax)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = _points(mol, n, n)
    _check(mol, pts, m.eval_esp(pts))


@pytest.mark.parametrize("n", [37887, 37889])
def test_two_points_per_thread(torch_cuda, n):
    mol = _molecule(2)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = _points(mol, n, n)
    _check(mol, pts, m.eval_esp(pts))


def test_results_do_not_depend_on_timing_and_nan_stays_with_its_point(torch_cuda):
    mol = _molecule(4)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = _points(mol, 1000, 5)
    a = m.eval_esp(pts)
    assert np.array_equal(a, m.eval_esp(pts))
    bad = pts.copy()
    bad[::100, 1] = np.nan
    bad[7] = 1e200
    b = m.eval_esp(bad)
    assert np.isnan(b[::100]).all()
    ok = np.ones(len(pts), bool)
    ok[::100] = ok[7] = False
    _check(mol, pts[ok], b[ok])
    assert abs(b[7]) < 1e-90
