"""The ESP at very distant points.  Where |P - C|^2 is finite (to 1e153 bohr) the
potential is that of the total charge, so r V(r) at 1e130 bohr equals r V(r) at
1e60 bohr; tolerance 1e-13 of the nuclear charge, rounding of a few hundred
terms.  Beyond, it is zero; at infinity it is zero with s functions alone and
NaN otherwise (the higher multipoles are infinity times zero)."""
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


def _molecule(lmax):
    rng = np.random.default_rng(lmax)
    coords = np.array([[0.0, 0.0, 0.0], [2.2, 0.4, -0.3], [-0.9, 1.9, 1.2]])
    shells = [S.Shell(center=coords[i % 3], atom=i % 3, angmoms=[am], exponents=np.array([0.3 * (i + 1)]),
                      coeffs=np.ones((1, 1))) for i, am in enumerate([0, 0, 0] + list(range(1, lmax + 1)))]
    M = sum(S.nfunc(a) for s in shells for a in s.angmoms)
    z = np.array([8.0, 6.0, 1.0])
    return S.SyntheticMolecule(coords=coords, numbers=z.astype(np.int32), charges=z, shells=shells,
                               D=S.make_density_matrix(rng, M, 2))


@pytest.mark.parametrize("n", [30, 300])  # one block and sorted points
@pytest.mark.parametrize("lmax", [0, 1, 4])
def test_distant_points(torch_cuda, lmax, n):
    mol = _molecule(lmax)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    rng = np.random.default_rng(n)
    base = mol.coords[rng.integers(0, 3, n)] + rng.normal(size=(n, 3))
    ref = m.eval_esp(base)
    pts = base.copy()
    inf = np.inf
    special = {0: [1e60, 0, 0], 1: [0, -1e130, 0], 2: [0, 0, 1e150], 3: [1e200, 1, 1], 4: [0, -1e308, 1e308],
               5: [inf, 0, 0], 6: [0, -inf, 2.0], 7: [-inf, inf, inf], 8: [np.nan, inf, 0], 9: [1e200, np.nan, 0]}
    for i, p in special.items():
        pts[i] = p
    got = m.eval_esp(pts)
    q = got[0] * 1e60
    for i, r in ((1, 1e130), (2, 1e150)):
        assert abs(got[i] * r - q) <= 1e-13 * mol.charges.sum(), (got[i] * r, q)
    assert (got[[3, 4]] == 0.0).all()
    if lmax == 0:
        assert (got[[5, 6, 7]] == 0.0).all()
    else:
        assert np.isnan(got[[5, 6, 7]]).all()
    assert np.isnan(got[[8, 9]]).all()
    assert np.allclose(got[10:], ref[10:], rtol=1e-12, atol=1e-13)
    np.testing.assert_array_equal(m.eval_esp_host(pts), got)
