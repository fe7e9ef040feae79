"""ctc_molecule_esp_info counts what the kernels cannot do without: every kept
pair in its far-field form.  One primitive per shell, so the kept pairs are the
shell pairs and their classes are known; and the rate that this count gives stays
below the FP64 pipe's 64 multiply-adds per clock and SM."""
import ctypes as C

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


def _far(L):
    return {0: 18, 1: 26}.get(L, 20 + (L + 1) * (L + 2) * (L + 3) // 3)


def _info(m):
    info = (C.c_double * 4)()
    ctc_abi.check(ctc_abi.lib().ctc_molecule_esp_info(m.h, info), "esp_info")
    return list(info)


def test_count_per_pair(torch_cuda):
    ls = [0, 0, 1, 2, 3, 4]
    coords = np.array([[0.0, 0.0, 0.0], [1.5, 0.2, -0.3]])
    shells = [S.Shell(center=coords[i % 2], atom=i % 2, angmoms=[l], exponents=np.array([0.5 + 0.1 * i]),
                      coeffs=np.ones((1, 1))) for i, l in enumerate(ls)]
    M = sum(S.nfunc(l) for l in ls)
    D = np.ones((M, M)) + np.eye(M)
    mol = S.SyntheticMolecule(coords=coords, numbers=np.array([6, 6], np.int32), charges=np.full(2, 6.0),
                              shells=shells, D=D)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pairs = [ls[i] + ls[j] for i in range(len(ls)) for j in range(i, len(ls))]
    info = _info(m)
    assert info[0] == len(pairs)
    assert info[1] == sum(_far(L) for L in pairs)
    assert info[3] == pytest.approx(np.mean(pairs))


def test_rate_is_below_the_pipe(torch_cuda):
    torch = torch_cuda
    mol = S.make_molecule("c5", seed=2, natom=40, box=13.0, nocc=80)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    n = 40_000
    pts = torch.as_tensor(S.random_points(np.random.default_rng(0), mol, n), device="cuda")
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    times = []
    for _ in range(4):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        ctc_abi.check(ctc_abi.lib().ctc_eval_esp(m.h, pts.data_ptr(), n, out.data_ptr(), None))
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e-3)
    p = torch.cuda.get_device_properties(0)
    peak = 2 * 64 * p.multi_processor_count * 1.98e9  # above the part's 1 965 MHz
    assert _info(m)[1] * n / min(times) < peak
