"""The ESP under a scratch limit (CTC_SCRATCH_LIMIT_BYTES): a call whose partial
sums and sorted points do not fit takes fewer slices, then fewer points at a
time, down to one row of partial sums per class and point (8 bytes each), which
is what a call needs at least.  Results as without a limit, up to the order of the
sums (1e-12 of the nuclear plus the electronic part)."""
import os

import numpy as np
import pytest

import ctc_abi
from test_gpu_esp_far import _molecule, _points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,n,limit", [(0, 100_000, 800_000), (0, 1_000, 8_000), (2, 200_000, 8_000_000),
                                          (2, 3_000, 120_000), (4, 5_000, 360_000)])
def test_limited_scratch(lmax, n, limit, monkeypatch):
    mol = _molecule(lmax)
    pts = _points(mol, n, 3)
    want = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D).eval_esp(pts)
    nuc = (mol.charges / np.linalg.norm(pts[:, None] - mol.coords[None], axis=-1)).sum(1)
    monkeypatch.setenv("CTC_SCRATCH_LIMIT_BYTES", str(limit))
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    for got in (m.eval_esp(pts), m.eval_esp_host(pts), m.eval_esp(pts)):
        assert (np.abs(got - want) <= 1e-12 * (nuc + np.abs(nuc - want))).all()


def test_no_room_at_all(monkeypatch):
    mol = _molecule(1)
    pts = _points(mol, 3000, 3)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    monkeypatch.setenv("CTC_SCRATCH_LIMIT_BYTES", "4096")
    assert os.environ["CTC_SCRATCH_LIMIT_BYTES"] == "4096"
    with pytest.raises(RuntimeError, match="-4: .*CTC_SCRATCH_LIMIT_BYTES"):
        m.eval_esp(pts)
    monkeypatch.delenv("CTC_SCRATCH_LIMIT_BYTES")
    assert np.isfinite(m.eval_esp(pts)).all()
