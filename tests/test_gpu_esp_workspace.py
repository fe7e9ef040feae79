"""The ESP's workspace when no pair is kept (a density matrix of zeros, such as
the spin density of a closed shell): points, sort buffers and keys alone, for
calls larger than the smallest block the workspace is given (1 MiB), against the
nuclear sum.  Tolerance: three terms, each a square root and a division of
rounded squares, 1e-14 of their sum.  Then the same molecule with pairs, whose
workspace is larger, and without again."""
import numpy as np
import pytest

import ctc_abi
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _molecule(D):
    coords = np.array([[0.0, 0.0, 0.0], [2.2, 0.4, -0.3], [-0.9, 1.9, 1.2]])
    z = np.array([8.0, 6.0, 1.0])
    shells = [S.Shell(center=coords[i], atom=i, angmoms=[0], exponents=np.array([0.9]), coeffs=np.ones((1, 1)))
              for i in range(3)]
    return S.SyntheticMolecule(coords=coords, numbers=z.astype(np.int32), charges=z, shells=shells, D=D)


@pytest.mark.parametrize("n", [1, 129, 20_000, 40_001, 300_000])
def test_no_pairs(torch_cuda, n):
    torch = torch_cuda
    mol = _molecule(np.zeros((3, 3)))
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = np.random.default_rng(n).uniform(-9.0, 9.0, (n, 3))
    nuc = (mol.charges / np.linalg.norm(pts[:, None] - mol.coords[None], axis=-1)).sum(1)
    np.testing.assert_allclose(m.eval_esp(pts), nuc, rtol=1e-14, atol=0)
    np.testing.assert_allclose(m.eval_esp_host(pts), nuc, rtol=1e-14, atol=0)
    for D in (np.eye(3), np.zeros((3, 3))):
        d = torch.as_tensor(D, device="cuda")
        ctc_abi.check(ctc_abi.lib().ctc_molecule_set_density_matrix(m.h, d.data_ptr(), None))
        got = m.eval_esp(pts)
        if D.any():
            assert (got < nuc).all()
        else:
            np.testing.assert_allclose(got, nuc, rtol=1e-14, atol=0)
