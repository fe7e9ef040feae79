"""A call that finds the device's memory taken fails with CTC_ERR_NOMEM and
leaves no error behind: once there is memory again, the next call succeeds with
correct results."""
import numpy as np
import pytest

import ctc_abi
from helpers import assert_close, term_scales
from oracle import oracle as O
from chemtoolscuda_b200 import synthetic as S

pytestmark = pytest.mark.gpu
KEYS = ("rho", "grad", "lap", "tau_pd")


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("precision,rtol", [(ctc_abi.PREC_FP64, 1e-10), (ctc_abi.PREC_TC, 1e-8)])
def test_recovery(torch_cuda, precision, rtol):
    torch = torch_cuda
    mol = S.make_molecule("c3", seed=5, natom=20, box=11.0, nocc=40)
    pts = S.random_points(np.random.default_rng(1), mol, 20_000, pad=2.0)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    m.eval_local(pts[:300], KEYS, precision)  # kernels loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = 48 << 20  # one tile per SM takes 145 MB
    fill = []
    for step in (1 << 30, 64 << 20, 8 << 20):
        while torch.cuda.mem_get_info()[0] > room + step:
            n = max(step, (torch.cuda.mem_get_info()[0] - room) // step * step) if step == 1 << 30 else step
            fill.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
    with pytest.raises(RuntimeError, match="-> -4: scratch allocation"):
        m.eval_local(pts, KEYS, precision)
    del fill
    torch.cuda.empty_cache()
    got = m.eval_local(pts, KEYS, precision)
    few = slice(0, 100)
    ref = O.eval_local(mol.flat(), mol.D, pts[few], alpha=0.5, keys=KEYS)
    sc = term_scales(mol.flat(), mol.D, pts[few], alpha=0.5)
    for k in KEYS:
        assert_close(k, got[k][few], ref[k], sc[k], rtol, atol=1e-15)
    assert m.sync_status() == 0
