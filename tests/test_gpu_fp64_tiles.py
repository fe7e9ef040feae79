"""The FP64 contraction at the edges of its tiles, slices and stages.

Basis sizes around the 32-function stages and 64-function slices, point counts
around the 32-, 64- and 128-point tiles (with few points the density runs on
32-point tiles, from 37 888 points on 128-point ones), a symmetric density
matrix (sums over the blocks on and above the diagonal) and one that is not
(full sums), against the same products formed in numpy from the oracle's AO
values.  Tolerance: the FP64 path's 1e-10 of the sum of absolute terms."""
import numpy as np
import pytest

import ctc_abi
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu
RTOL = 1e-10
HESS = {(0, 0): 4, (0, 1): 5, (0, 2): 6, (1, 1): 7, (1, 2): 8, (2, 2): 9}


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _molecule(M, symmetric=True):
    """M functions (p shells, then s shells for the rest) on five atoms."""
    rng = np.random.default_rng(M)
    coords = np.array([[0, 0, 0], [1.9, 0.3, -0.4], [-1.2, 1.6, 0.8], [0.4, -1.7, 1.3], [1.1, 1.2, 2.0]], float)
    shells, left = [], M
    while left:
        am = 1 if left >= 8 else 0
        a = len(shells) % 5
        e = np.exp(rng.uniform(np.log(0.15), np.log(20.0), size=2))
        shells.append(S.Shell(center=coords[a], atom=a, angmoms=[am], exponents=e, coeffs=rng.standard_normal((1, 2))))
        left -= S.nfunc(am)
    D = S.make_density_matrix(rng, M, max(1, M // 3))
    if not symmetric:
        D = D + 0.1 * np.abs(D).max() * rng.standard_normal(D.shape)
    return S.SyntheticMolecule(coords=coords, numbers=np.full(5, 6), charges=np.full(5, 6.0), shells=shells, D=D)


def _reference(mol, pts):
    A = O.eval_ao(mol.flat(), pts, 2)
    out = []
    for a, d in ((A, mol.D), (np.abs(A), np.abs(mol.D))):
        G = [a[q] @ d for q in range(4)]
        v = dict(rho=(G[0] * a[0]).sum(1), grad=2 * np.stack([(G[0] * a[1 + k]).sum(1) for k in range(3)], 1),
                 tau_pd=0.5 * sum((G[1 + k] * a[1 + k]).sum(1) for k in range(3)), hess=np.zeros((len(pts), 3, 3)))
        for (i, j), q in HESS.items():
            v["hess"][:, i, j] = v["hess"][:, j, i] = 2 * ((G[1 + i] * a[1 + j]).sum(1) + (G[0] * a[q]).sum(1))
        v["lap"] = np.trace(v["hess"], axis1=1, axis2=2)
        out.append(v)
    return out


def _check(got, ref, scale):
    for k, x in got.items():
        assert np.isfinite(x).all(), k
        assert (np.abs(x - ref[k]) <= RTOL * scale[k] + 1e-15).all(), (k, np.abs(x - ref[k]).max())


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("M", [1, 31, 32, 33, 64, 65, 96, 97, 161, 200])
def test_local_sizes(torch_cuda, M, symmetric):
    mol = _molecule(M, symmetric)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    for n in (1, 31, 33, 129):
        pts = S.random_points(np.random.default_rng(n), mol, n, pad=2.0)
        ref, scale = _reference(mol, pts)
        for keys in (("rho",), ("rho", "grad"), ("rho", "tau_pd"), ("rho", "grad", "hess", "lap", "tau_pd")):
            _check(m.eval_local(pts, keys), ref, scale)


@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("n", [37887, 37888, 40001])
def test_density_tile_sizes(torch_cuda, n, symmetric):
    mol = _molecule(70, symmetric)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = S.random_points(np.random.default_rng(n), mol, n, pad=2.0)
    ref, scale = _reference(mol, pts)
    for keys in (("rho",), ("rho", "grad")):
        _check(m.eval_local(pts, keys), ref, scale)


def test_symmetry_follows_the_density_matrix(torch_cuda):
    """The full sums are taken as soon as D is replaced by one that is not symmetric, and back."""
    torch = torch_cuda
    mol, skew = _molecule(97), _molecule(97, symmetric=False)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = S.random_points(np.random.default_rng(3), mol, 70, pad=2.0)
    for x in (mol, skew, mol):
        d = torch.as_tensor(x.D, device="cuda")
        ctc_abi.check(ctc_abi.lib().ctc_molecule_set_density_matrix(m.h, d.data_ptr(), None))
        ref, scale = _reference(x, pts)
        _check(m.eval_local(pts, ("rho", "grad", "hess", "tau_pd")), ref, scale)
        _check(m.eval_local(pts, ("rho",)), ref, scale)


@pytest.mark.parametrize("with_grad", [True, False])
@pytest.mark.parametrize("M,n", [(1, 1), (33, 63), (64, 64), (65, 65), (97, 129), (161, 300)])
def test_adjoint_sizes(torch_cuda, M, n, with_grad):
    mol = _molecule(M)
    rng = np.random.default_rng(M + n)
    pts = S.random_points(rng, mol, n, pad=2.0)
    vr = rng.standard_normal(n)
    vg = rng.standard_normal((n, 3)) if with_grad else None
    vr[::3] = 0.0  # points with zero weight
    if vg is not None:
        vg[::3] = 0.0
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    rD, rR = O.adjoint(mol.flat(), mol.D, len(mol.coords), pts, vr, vg)
    for want_D, want_R in ((True, True), (True, False), (False, True)):
        dD, dR = m.adjoint(pts, vr, vg, want_D=want_D, want_R=want_R)
        if want_D:
            np.testing.assert_allclose(dD, rD, rtol=0, atol=RTOL * np.abs(rD).max() + 1e-15)
        if want_R:
            np.testing.assert_allclose(dR, rR, rtol=0, atol=RTOL * np.abs(rR).max() + 1e-15)
