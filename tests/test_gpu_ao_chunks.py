"""AO values at few points (chunks of 32 functions, on more CTAs) and at more
(chunks of 64): bases whose chunks end within and at a segment, one point to past
the line, every derivative order.  Against the FP64 oracle, 1e-12 of each
quantity's largest value (a contraction of at most six primitives)."""
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


@pytest.mark.parametrize("config,natom", [("c1", 2), ("c4", 6), ("c2", 30)])
@pytest.mark.parametrize("n", [1, 32, 33, 500, 2500])
def test_values_and_derivatives(torch_cuda, config, natom, n):
    mol = S.make_molecule(config, seed=natom, natom=natom, box=3.0 * natom ** (1 / 3) + 1.5, nocc=2)
    pts = S.random_points(np.random.default_rng(n), mol, n, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    for deriv in (0, 1, 2):
        got, ref = m.eval_ao(pts, deriv), O.eval_ao(mol.flat(), pts, deriv)
        for q in range(got.shape[0]):
            assert np.isfinite(got[q]).all()
            np.testing.assert_allclose(got[q], ref[q], rtol=0, atol=1e-12 * np.abs(ref[q]).max())
