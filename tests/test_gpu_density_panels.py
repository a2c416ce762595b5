"""The unfactored staged contraction at basis sizes whose output panels are not a multiple of 32
columns wide before rounding (kpad 704, 832 and 960: 235, 208 and 240 columns a panel)."""
import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from qmtools import synthetic as syn
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms,kpad", [(66, 704), (80, 832), (91, 960)])
def test_every_panel_column_counts(basis, natoms, kpad):
    rng = np.random.default_rng(natoms)
    types = syn.element_list(natoms, rng)
    side = syn.cube_side(natoms)
    xyz = syn.random_geometry(natoms, side, rng)
    n = sum(14 if z > 1 else 5 for z in types)
    assert kpad - 64 < n <= kpad
    a = rng.standard_normal((n, n)) / n
    dm = a @ a.T + 0.01 * np.diag(rng.random(n))     # full rank: the unfactored contraction
    rows = [[int(z), *(float(v) for v in p / syn.ANG2BOR)] for z, p in zip(types, xyz)]
    mol = qmtools.Molecule(rows, dm, basis)
    g = qmtools.Grid((1, 16, 16, 16), side / 16 / qmtools.ANG2BOR, [0.01, 0.02, 0.03])
    ref = qmtools.QMTools.Compute_density(g, mol, precision="fp64", rescale=False).qube.ravel()
    N.call("qmt_set_density_path", 1)
    try:
        got = qmtools.QMTools.Compute_density(g, mol, precision="fp16x3", rescale=False).qube.ravel()
    finally:
        N.call("qmt_set_density_path", 0)
    # kpad / 16 K-steps of three products, each FP32 addition off by at most 2^-23 of the sum
    assert rel_l2(got, ref) <= 3 * kpad / 16 * 2.0 ** -23
    mol.release()
