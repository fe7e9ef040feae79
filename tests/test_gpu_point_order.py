"""Explicit points on molecules of every length the ordering rules tell apart
(unsorted, 24-bit and 30-bit Morton keys; chemtoolscuda_b200/csrc/ctc_chunk.h),
with non-finite points among them: every point's result is its own, whatever the
order.  Against the FP64 oracle, 1e-10 (FP64) and 1e-8 (tensor cores) of the sum
of absolute terms; the ESP 1e-12 of the nuclear plus the electronic part, and
1e-10 for the pairs it drops (their bounds sum to 1e-11) and its oracle."""
import ctypes as C

import numpy as np
import pytest

import ctc_abi
from helpers import assert_close, term_scales
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu
KEYS = ("rho", "grad", "lap", "tau_pd")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _chain(natom, step):
    rng = np.random.default_rng(natom)
    coords = np.zeros((natom, 3))
    coords[:, 0] = np.arange(natom) * step
    coords += rng.normal(scale=0.3, size=coords.shape)
    z = rng.choice([1, 6, 8], size=natom)
    shells = S.make_basis(rng, coords, z, S.RECIPES["c1"])
    M = sum(S.nfunc(a) for s in shells for a in s.angmoms)
    return S.SyntheticMolecule(coords=coords, numbers=z.astype(np.int32), charges=z.astype(float), shells=shells,
                               D=S.make_density_matrix(rng, M, max(1, M // 4)))


def _noalloc(torch, m, pts):
    L = ctc_abi.lib()
    L.ctc_eval_local_noalloc.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    d = torch.as_tensor(pts, device="cuda")
    rho = torch.full((len(pts),), float("nan"), dtype=torch.float64, device="cuda")
    o = ctc_abi.Outputs(rho=rho.data_ptr())
    ctc_abi.check(L.ctc_eval_local_noalloc(m.h, d.data_ptr(), len(pts), None, C.byref(o), None), "noalloc")
    torch.cuda.synchronize()
    return rho.cpu().numpy()


# length + 24 bohr: 34 (24 bits, unsorted when small), 144 (sorted when small too), 534 and 1 224 (30 bits)
@pytest.mark.parametrize("natom,step", [(6, 2.0), (13, 10.0), (18, 30.0), (25, 50.0)])
@pytest.mark.parametrize("n", [40, 300, 2048, 2049])
def test_every_order(torch_cuda, natom, step, n):
    mol = _chain(natom, step)
    rng = np.random.default_rng(n)
    pts = mol.coords[rng.integers(0, natom, n)] + rng.normal(scale=1.5, size=(n, 3))
    bad = np.zeros(n, bool)
    bad[[3, n // 2, n - 1]] = True
    pts[3, 0], pts[n // 2, 1], pts[n - 1] = np.nan, np.inf, -np.inf
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    few = np.flatnonzero(~bad)[:: max(1, n // 200)]
    ref = O.eval_local(mol.flat(), mol.D, pts[few], alpha=0.5, keys=KEYS)
    sc = term_scales(mol.flat(), mol.D, pts[few], alpha=0.5)
    for precision, rtol in ((ctc_abi.PREC_FP64, 1e-10), (ctc_abi.PREC_TC, 1e-8)):
        got = m.eval_local(pts, KEYS, precision)
        for k in KEYS:
            assert np.isnan(got[k][bad]).all() and np.isfinite(got[k][~bad]).all()
            assert_close(k, got[k][few], ref[k], sc[k], rtol, atol=1e-15)
    rho = _noalloc(torch_cuda, m, pts)
    assert np.isnan(rho[bad]).all()
    assert_close("rho", rho[few], ref["rho"], sc["rho"], 1e-10, atol=1e-15)
    assert m.sync_status() == 0
    few = few[:40]
    v = m.eval_esp(pts)
    want = O.eval_esp(mol.flat(), mol.D, mol.coords, mol.charges, pts[few])
    nuc = (mol.charges / np.linalg.norm(pts[few][:, None] - mol.coords[None], axis=-1)).sum(1)
    assert (np.abs(v[few] - want) <= 1e-12 * (nuc + np.abs(nuc - want)) + 1e-10).all()
    assert np.isnan(v[3]) and np.isfinite(v[~bad]).all()
