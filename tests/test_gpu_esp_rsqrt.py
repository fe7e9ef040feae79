"""The reciprocal square root of the ESP's far-field sum (esp_rsqrt, an
approximation and one Householder step; ctc_esp.cu) over the range of |P - C|^2
it is used in, through the potential of one s function at the origin without a
nucleus: V(r) = -q / r for points on the axes, where |P - C|^2 is r^2 rounded
once.  r V(r) is the same number everywhere up to the rounding of r^2 (2^-54 of
the root), the root (1.4e-16, as stated there) and the final multiply-add
(2^-53): 3.1e-16 together; the reference is the median, off by at most as much.
Formed in long double."""
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


@pytest.mark.parametrize("lo,hi", [(1e-2, 1.0), (1.0, 64.0), (64.0, 1e9), (1e9, 1e150)])
def test_relative_error(torch_cuda, lo, hi):
    # T = 2 a r^2 >= 38 from r = 1e-2 on: every pair is a far pair
    sh = S.Shell(center=np.zeros(3), atom=0, angmoms=[0], exponents=np.array([1e6]), coeffs=np.ones((1, 1)))
    mol = S.SyntheticMolecule(coords=np.zeros((1, 3)), numbers=np.array([1], np.int32), charges=np.zeros(1),
                              shells=[sh], D=np.ones((1, 1)))
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    rng = np.random.default_rng(7)
    n = 300_000
    r = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    pts = np.zeros((n, 3))
    pts[np.arange(n), rng.integers(0, 3, n)] = r * rng.choice([-1.0, 1.0], n)
    rv = m.eval_esp(pts).astype(np.longdouble) * r.astype(np.longdouble)
    q = np.median(rv)
    assert q < 0
    worst = np.abs(rv / q - 1).max()
    assert worst <= 2 * 3.1e-16, float(worst)
