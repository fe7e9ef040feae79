"""Every class of primitive pairs up to g-g in the ESP's far- and near-field
polynomials, tightly: 1e-12 of the nuclear plus the electronic part (rounding of
a few thousand terms of either sign), and 1e-11, the bound of the pairs that are
dropped.  Points from 0.3 to 200 bohr from a nucleus, against the FP64 oracle."""
import numpy as np
import pytest

import ctc_abi
from oracle import oracle as O
from test_gpu_esp_far import _molecule, _points

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [90, 700])
@pytest.mark.parametrize("lmax", [0, 1, 2, 3, 4])
def test_classes(lmax, n):
    mol = _molecule(lmax)
    m = ctc_abi.Mol(mol.flat(), mol.coords, mol.charges, mol.D)
    pts = _points(mol, n, 100 + n)
    ref = O.eval_esp(mol.flat(), mol.D, mol.coords, mol.charges, pts)
    nuc = (mol.charges / np.linalg.norm(pts[:, None] - mol.coords[None], axis=-1)).sum(1)
    got = m.eval_esp(pts)
    assert (np.abs(got - ref) <= 1e-12 * (nuc + np.abs(nuc - ref)) + 1e-11).all(), np.abs(got - ref).max()
