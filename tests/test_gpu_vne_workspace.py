"""The pseudo-field keeps out of the workspace that an FFT solve captured in a graph goes on reading."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from qmtools import synthetic as syn

pytestmark = pytest.mark.gpu


def test_captured_solve_survives_a_larger_pseudo_field(basis):
    import torch
    sm = syn.config_molecule("c0")
    mol = sm.molecule(basis, qmtools.Molecule)
    N.ensure_device()
    n, h = 16, 0.7
    org = [float(o) for o in np.asarray(sm.coords_bohr).mean(axis=0) - n * h / 2]
    q = torch.rand(n ** 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    v = torch.empty_like(q)

    def solve():
        N.call("qmt_fft_poisson", mol.handle, n, n, n, h, *org, 0.2, 6.0, 0, C.c_void_p(q.data_ptr()),
               C.c_void_p(v.data_ptr()), N.stream_handle())

    solve()
    torch.cuda.synchronize()
    ref = v.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        solve()
    big = (64, 64, 64)
    res, out = (torch.empty(int(np.prod(big)), device="cuda") for _ in range(2))
    it = C.c_int()
    N.call("qmt_vne_pseudo", mol.handle, *big, 0.2, *org, 0.05, 0.02, 1e-12, 2, C.c_void_p(res.data_ptr()),
           C.c_void_p(out.data_ptr()), C.byref(it), N.stream_handle())
    v.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(v, ref)
    mol.release()
