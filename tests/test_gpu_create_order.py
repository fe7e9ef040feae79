"""A molecule is complete when ctc_molecule_create returns: its first evaluation,
on a non-blocking stream (which is not ordered behind the default stream), sees
the symmetry flag of its density matrix.  A matrix that is not symmetric only in
its last function's row takes the full sums; the half sums would be off by that
row's asymmetry.  rho against the same product in numpy from the oracle's AO
values, at the FP64 path's 1e-10 of the sum of absolute terms."""
import ctypes as C

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


def test_first_call_on_a_non_blocking_stream(torch_cuda):
    torch = torch_cuda
    mol = S.make_molecule("c2", seed=3, natom=150, box=22.0, nocc=40)
    M = mol.nbasis
    rng = np.random.default_rng(4)
    D = mol.D.copy()
    D[M - 1] += 0.5 * np.abs(D).max() * rng.standard_normal(M)
    pts = np.ascontiguousarray(mol.shells[-1].center + rng.uniform(-1.0, 1.0, (40, 3)))
    phi = O.eval_ao(mol.flat(), pts, 0)[0]
    ref = ((phi @ D) * phi).sum(1)
    scale = ((np.abs(phi) @ np.abs(D)) * np.abs(phi)).sum(1)
    half = ((phi @ (np.triu(D) + np.triu(D, 1).T)) * phi).sum(1)
    assert (np.abs(half - ref) > 1e-6 * scale).any(), "the asymmetry must show"
    side = torch.cuda.Stream()
    for _ in range(8):
        d_pts = torch.as_tensor(pts, device="cuda")
        rho = torch.empty(len(pts), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, D)
        o = ctc_abi.Outputs(rho=rho.data_ptr())
        ctc_abi.check(ctc_abi.lib().ctc_eval_local(m.h, d_pts.data_ptr(), len(pts), ctc_abi.PREC_FP64, None,
                                                   C.byref(o), side.cuda_stream), "ctc_eval_local")
        side.synchronize()
        assert (np.abs(rho.cpu().numpy() - ref) <= 1e-10 * scale).all()
        got = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, D).eval_local_host(pts, ("rho",))["rho"]
        assert (np.abs(got - ref) <= 1e-10 * scale).all()
        m.close()
