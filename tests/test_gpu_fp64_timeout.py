"""Bounded waits of the FP64 contraction that run out: the molecule's wait limit
is cut to one SM cycle, so that the waits of its loaders, matrix warps and
epilogue give up at once.  The kernel must stop, wait for its own copies in
flight and record CTC_ERR_DEVICE; with the limit restored the molecule gives
correct results again.  Every form of the kernel: four rows per point, phi rows
on small and on large tiles, and the two force forms."""
import os
import sys

import numpy as np
import pytest

import ctc_abi
from helpers import assert_close, term_scales
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))

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
