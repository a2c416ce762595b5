"""The SIMT density kernel at every panel width its dispatch picks (one panel of 64 to 256 columns, P held in
shared memory or read in chunks, two and three panels), against the FP64 oracle with the tolerances of
the density tests."""
import numpy as np
import pytest

import qmtools
from oracle import density as od
from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-7, "fp32": 1e-6}


@pytest.mark.parametrize("heavy,light", [(0, 3), (2, 4), (5, 3), (8, 2), (10, 3), (12, 2), (15, 2), (18, 0), (20, 2),
                                         (26, 0), (40, 1)])
@pytest.mark.parametrize("prec,sub", [("fp64", 1), ("fp32", 1), ("fp64", 3)])
def test_panel_widths(basis, heavy, light, prec, sub):
    rng = np.random.default_rng(heavy)
    zs = [6] * heavy + [1] * light
    k = int(np.ceil(len(zs) ** (1 / 3)))
    pos = np.array([(x, y, z) for x in range(k) for y in range(k) for z in range(k)][:len(zs)]) * 1.3
    rows = [[z, *(float(v) for v in p)] for z, p in zip(zs, pos)]
    n = 14 * heavy + 5 * light
    a = rng.standard_normal((n, n)) / n
    mol = qmtools.Molecule(rows, a @ a.T, basis)
    c = np.asarray(mol.coords).mean(axis=0)
    g = qmtools.Grid((1, 8, 8, 8), 0.7 / qmtools.ANG2BOR, list(c - 2.8 + 0.01))
    nx, ny, nz, h, ox, oy, oz = g._geom()
    ref = od.density_qube_unscaled((nx, ny, nz), np.float32(h), (ox, oy, oz), mol.coords, mol.ALMOs, basis.alphas,
                                   basis.coeffs, mol.dm, sub)
    got = qmtools.QMTools.Compute_density(g, mol, subgrid=sub, precision=prec, rescale=False).qube.ravel()
    assert rel_l2(got, ref) <= TOL[prec]
    mol.release()
