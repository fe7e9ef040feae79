"""ctc_molecule_set_density_matrix: the library's copy in its own order and the
symmetry flag come from one pass over 32 x 32 blocks and their mirror images.
Basis sizes around the blocks and the padding, and matrices that are symmetric but
for one element: near the diagonal, in a corner, in the first and the last block.
rho (half sums with a symmetric matrix, full sums otherwise) against numpy with
the oracle's AO values at the FP64 path's 1e-10; the ESP, which reads the copy
back, against a molecule created with the same matrix, to the last bit."""
import numpy as np
import pytest

import ctc_abi
from chemtoolscuda_b200 import synthetic as S
from oracle import oracle as O
from test_gpu_fp64_tiles import _molecule

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("M", [1, 2, 31, 32, 33, 127, 128, 129, 200])
def test_copy_and_flag(torch_cuda, M):
    torch = torch_cuda
    mol = _molecule(M)
    rng = np.random.default_rng(M)
    pts = S.random_points(rng, mol, 50, pad=1.0)
    phi = O.eval_ao(mol.flat(), pts, 0)[0]
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, np.zeros((M, M)))
    skew = {(M - 1, 0), (0, M - 1), (M // 2, M // 2 - 1), (M - 1, M - 2), (min(31, M - 1), min(32, M - 1)), (1, 0)}
    for at in [None] + sorted(p for p in skew if p[0] != p[1] and min(p) >= 0 and max(p) < M) + [None]:
        D = S.make_density_matrix(rng, M, max(1, M // 3))
        if at is not None:
            D[at] += 0.7 * np.abs(D).max()
        d = torch.as_tensor(D, device="cuda")
        ctc_abi.check(ctc_abi.lib().ctc_molecule_set_density_matrix(m.h, d.data_ptr(), None))
        got = m.eval_local(pts, ("rho",))["rho"]
        ref = ((phi @ D) * phi).sum(1)
        assert (np.abs(got - ref) <= 1e-10 * ((np.abs(phi) @ np.abs(D)) * np.abs(phi)).sum(1) + 1e-15).all(), at
        fresh = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, D)
        np.testing.assert_array_equal(m.eval_esp(pts), fresh.eval_esp(pts))
        np.testing.assert_array_equal(got, fresh.eval_local(pts, ("rho",))["rho"])
