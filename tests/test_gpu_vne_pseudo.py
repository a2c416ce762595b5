"""The pseudo-field's sweeps in one launch: rows of four points and single points (nx not a multiple of 4),
grids without inner points, pair counts, against the FP64 oracle (its tolerance for this field, 1e-5)."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from qmtools import synthetic as syn
from oracle import gridops as og
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 24, 8), (13, 9, 11), (4, 5, 6), (2, 7, 7), (1, 1, 1), (40, 33, 20)])
@pytest.mark.parametrize("iters", [0, 5])
def test_matches_oracle(basis, shape, iters):
    import torch
    sm = syn.config_molecule("c0")
    mol = sm.molecule(basis, qmtools.Molecule)
    nx, ny, nz = shape
    h = 0.7
    o = (np.asarray(sm.coords_bohr).mean(axis=0) - np.array(shape) * h / 2).astype(np.float32)
    n = nx * ny * nz
    res = torch.full((n + 32,), 5.0, device="cuda")
    out = torch.full((n + 32,), 5.0, device="cuda")
    it = C.c_int()
    N.call("qmt_vne_pseudo", mol.handle, nx, ny, nz, h, float(o[0]), float(o[1]), float(o[2]), 0.05, 0.02, 1e-12, iters,
           C.c_void_p(res.data_ptr()), C.c_void_p(out.data_ptr()), C.byref(it), N.stream_handle())
    ref, pairs = og.vne_pseudo(shape, np.float32(h), tuple(float(v) for v in o), mol.coords, mol.types, ads=0.05, dif=0.02,
                               tolerance=1e-12, maxiters=iters)
    got = res.cpu().numpy()
    assert it.value == pairs
    assert np.all(got[n:] == 5.0)
    if np.any(ref):
        assert rel_l2(got[:n], ref) <= 1e-5
    else:
        assert not np.any(got[:n])
    mol.release()
