"""Bounded waits of the FP64 contraction that run out: the molecule's wait limit
is cut to one SM cycle, so that the waits of its loaders, matrix warps and
epilogue give up at once.  The kernel must stop, wait for its own copies in
flight and record CTC_ERR_DEVICE; with the limit restored the molecule gives
correct results again.  Every form of the kernel: four rows per point, phi rows
on small and on large tiles, and the two force forms."""
import ctypes as C

import numpy as np
import pytest

import ctc_abi
from helpers import assert_close, term_scales
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(scope="module")
def molecule():
    return S.make_molecule("c3", seed=5, natom=20, box=11.0, nocc=40)


def _check(mol, pts, got, keys):
    few = slice(0, 100)
    ref = O.eval_local(mol.flat(), mol.D, pts[few], alpha=0.5, keys=keys)
    sc = term_scales(mol.flat(), mol.D, pts[few], alpha=0.5)
    for k in keys:
        assert_close(k, got[k][few], ref[k], sc[k], 1e-10, atol=1e-15)


@pytest.mark.parametrize("n,keys", [(3000, ("rho", "grad", "hess", "tau_pd")), (3000, ("rho",)),
                                    (40_000, ("rho",)), (40_000, ("rho", "grad"))])
def test_local(torch_cuda, molecule, n, keys):
    mol = molecule
    pts = S.random_points(np.random.default_rng(n), mol, n, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    m.set_wait_limit(1)
    for _ in range(3):
        m.eval_local(pts, keys)  # stream-ordered: returns CTC_OK
        assert m.sync_status() == -5, "a one-cycle wait limit must run out"
        assert "FP64 contraction" in ctc_abi.err()
        assert m.sync_status() == 0  # reporting clears the record
    with pytest.raises(RuntimeError, match="FP64 contraction"):
        m.eval_local_host(pts, keys)  # waits, so it reports its own failure
    m.set_wait_limit(0)
    _check(mol, pts, m.eval_local(pts, keys), keys)
    assert m.sync_status() == 0
    m.close()


@pytest.mark.parametrize("with_grad", [True, False])
def test_adjoint(torch_cuda, molecule, with_grad):
    """The adjoint records its own failure, and its next call reports it."""
    mol = molecule
    rng = np.random.default_rng(8)
    n = 3000
    pts = S.random_points(rng, mol, n, pad=2.0)
    vr, vg = rng.standard_normal(n), rng.standard_normal((n, 3)) if with_grad else None
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    m.set_wait_limit(1)
    m.adjoint(pts, vr, vg)
    assert m.sync_status() == -5
    assert "FP64 contraction" in ctc_abi.err()
    m.adjoint(pts, vr, vg)
    m.set_wait_limit(0)
    with pytest.raises(RuntimeError, match="earlier call.*FP64 contraction"):
        m.adjoint(pts, vr, vg)
    few = slice(0, 60)
    dD, dR = m.adjoint(pts[few], vr[few], None if vg is None else vg[few])
    rD, rR = O.adjoint(mol.flat(), mol.D, len(mol.coords), pts[few], vr[few], None if vg is None else vg[few])
    np.testing.assert_allclose(dD, rD, rtol=0, atol=1e-10 * np.abs(rD).max())
    np.testing.assert_allclose(dR, rR, rtol=0, atol=1e-10 * np.abs(rR).max())
    assert m.sync_status() == 0
    m.close()


def _noalloc(torch, m, d_pts, rho, tau):
    L = ctc_abi.lib()
    L.ctc_eval_local_noalloc.argtypes = [C.c_void_p, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p]
    o = ctc_abi.Outputs(rho=rho.data_ptr(), tau_pd=tau.data_ptr())
    ctc_abi.check(L.ctc_eval_local_noalloc(m.h, d_pts.data_ptr(), d_pts.shape[0], None, C.byref(o),
                                           torch.cuda.current_stream().cuda_stream), "ctc_eval_local_noalloc")


def test_noalloc(torch_cuda, molecule):
    """The call without allocations does the same; captured into a graph it leaves
    the status to ctc_molecule_sync_status and later calls as they were."""
    torch, mol = torch_cuda, molecule
    pts = S.random_points(np.random.default_rng(2), mol, 2000, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    d = torch.as_tensor(pts, device="cuda")
    rho, tau = (torch.full((len(pts),), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2))
    m.set_wait_limit(1)
    _noalloc(torch, m, d, rho, tau)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="earlier call.*FP64 contraction"):
        _noalloc(torch, m, d, rho, tau)
    m.set_wait_limit(0)
    _noalloc(torch, m, d, rho, tau)
    torch.cuda.synchronize()
    want = rho.clone(), tau.clone()
    _check(mol, pts, {"rho": rho.cpu().numpy(), "tau_pd": tau.cpu().numpy()}, ("rho", "tau_pd"))
    assert m.sync_status() == 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _noalloc(torch, m, d, rho, tau)
    for _ in range(2):
        rho.fill_(float("nan"))
        tau.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(rho, want[0]) and torch.equal(tau, want[1])
        got = m.eval_local(pts, ("rho", "tau_pd"))
        _check(mol, pts, got, ("rho", "tau_pd"))
    assert m.sync_status() == 0
    m.close()
