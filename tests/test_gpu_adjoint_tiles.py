"""The adjoint's tiles of 32 and of 64 points (few and many points per SM): edges
of both, and the line between them (32 points per SM; 4 736 on 148), on molecules
whose points keep most functions and on a chain where tiles keep different ones.
Against the FP64 oracle, 1e-10 of the largest entry."""
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


def _chain(natom, step):
    rng = np.random.default_rng(natom)
    coords = np.zeros((natom, 3))
    coords[:, 0] = np.arange(natom) * step
    z = rng.choice([1, 6], size=natom)
    shells = S.make_basis(rng, coords, z, S.RECIPES["c2"])
    M = sum(S.nfunc(a) for s in shells for a in s.angmoms)
    return S.SyntheticMolecule(coords=coords, numbers=z.astype(np.int32), charges=z.astype(float), shells=shells,
                               D=S.make_density_matrix(rng, M, max(1, M // 4)))


@pytest.mark.parametrize("step", [1.5, 12.0])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 1000, "line", "line+1"])
def test_tiles(torch_cuda, step, n):
    sms = torch_cuda.cuda.get_device_properties(0).multi_processor_count
    n = {"line": 32 * sms, "line+1": 32 * sms + 1}.get(n, n)
    mol = _chain(9, step)
    rng = np.random.default_rng(n)
    pts = mol.coords[rng.integers(0, 9, n)] + rng.normal(scale=1.5, size=(n, 3))
    vr, vg = rng.standard_normal(n), rng.standard_normal((n, 3))
    vr[::5] = 0.0
    vg[::5] = 0.0
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    rD, rR = O.adjoint(mol.flat(), mol.D, 9, pts, vr, vg)
    for want_D in (True, False):
        dD, dR = m.adjoint(pts, vr, vg, want_D=want_D)
        np.testing.assert_allclose(dR, rR, rtol=0, atol=1e-10 * np.abs(rR).max())
        if want_D:
            np.testing.assert_allclose(dD, rD, rtol=0, atol=1e-10 * np.abs(rD).max())
    assert m.sync_status() == 0
