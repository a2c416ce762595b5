"""The factored contraction's uniform loss, without the rescaling that hides it, at one, two and three accumulators
of the large products (ranks up to 64, up to 80 and above).

The tensor core's FP32 additions truncate: each of the n K-steps summed in one accumulator takes at most 2^-23 of
it, half of that on average, and the squares double the loss, so the grid total falls by about n 2^-23 at most;
the factor, the split and the FP32 basis functions add at most 2e-7 between them.
"""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from qmtools import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("config,rank", [("c0", 1), ("c0", 9), ("c1", 16), ("c1", 59), ("c1", 64), ("c1", 72),
                                         ("c1", 90), ("c1", 110)])
def test_uniform_loss(basis, config, rank):
    import torch
    N.ensure_device()
    sm = syn.config_molecule(config)
    mol = sm.molecule(basis, qmtools.Molecule)
    n = int(mol.norbs)
    g = np.random.default_rng(rank)
    c = np.linalg.qr(g.standard_normal((n, rank)))[0]
    mol.set_dm((c @ c.T).astype(np.float32))
    shape, h = (40, 40, 40), 0.7
    org = [float(o) for o in np.asarray(sm.coords_bohr).mean(axis=0) - np.array(shape) * h / 2]
    q = torch.empty(int(np.prod(shape)), device="cuda")
    out = {}
    for prec in ("fp64", "fp16x3"):
        s = C.c_double()
        N.call("qmt_density", mol.handle, *shape, h, *org, 1, N.PREC[prec], 0, C.c_void_p(q.data_ptr()), C.byref(s),
               N.stream_handle())
        out[prec] = q.double().sum().item()
    r = C.c_int()
    N.call("qmt_density_factor_rank", mol.handle, C.byref(r), N.stream_handle())
    assert r.value >= rank
    units = -(-n // 10)   # of 16 columns, at least ten of them filled
    na = max(1, min(3, 256 // (-(-r.value // 16) * 16) - 1))
    assert abs(out["fp16x3"] / out["fp64"] - 1) < -(-units // na) * 2.0 ** -23 + 2e-7
