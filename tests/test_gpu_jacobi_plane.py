"""The plane Jacobi kernel (one CTA per plane) against the grid-barrier kernel: identical grids and sweep
counts at the edges of its range -- one group of points per thread up to four, partly filled last groups, rows
that straddle warps, few and many planes -- and its convergence stop and give-up path."""
import ctypes as C

import pytest

from qmtools import _native as N

pytestmark = pytest.mark.gpu


def _solve(fn, shape, sweeps, path, tol=0.0, every=7):
    import torch
    N.ensure_device()
    n = shape[0] * shape[1] * shape[2]
    g = torch.Generator(device="cuda").manual_seed(11)
    rho = torch.rand(n, device="cuda", generator=g) - 0.5
    v = torch.rand(n, device="cuda", generator=g)
    t = torch.full_like(v, 3.0)
    sw, dl = C.c_int(), C.c_double()
    N.call("qmt_set_jacobi_path", path)
    try:
        st = getattr(N.load(), fn)(*shape, C.c_float(0.2), C.c_void_p(rho.data_ptr()), C.c_void_p(v.data_ptr()),
                                   C.c_void_p(t.data_ptr()), sweeps, every, tol, C.byref(sw), C.byref(dl),
                                   N.stream_handle())
    finally:
        N.call("qmt_set_jacobi_path", 0)
    return st, sw.value, dl.value, v


@pytest.mark.parametrize("fn", ["qmt_jacobi", "qmt_jacobi_dirichlet"])
@pytest.mark.parametrize("shape", [(64, 64, 64), (36, 40, 33), (4, 128, 80), (120, 56, 56), (132, 100, 50),
                                   (128, 128, 128), (128, 124, 148), (48, 3, 300)])
def test_identical_to_grid_barrier_kernel(fn, shape):
    import torch
    a = _solve(fn, shape, 30, 0)
    b = _solve(fn, shape, 30, 1)
    assert a[:2] == b[:2] == (N.OK, 30)
    assert torch.equal(a[3], b[3])
    assert a[2] == pytest.approx(b[2], rel=1e-12)      # the residual's order of summation differs


def test_stops_at_tolerance_like_grid_barrier_kernel():
    import torch
    ref = _solve("qmt_jacobi_dirichlet", (64, 64, 48), 40, 1)
    a = _solve("qmt_jacobi_dirichlet", (64, 64, 48), 400, 0, tol=ref[2] * 1.2)
    b = _solve("qmt_jacobi_dirichlet", (64, 64, 48), 400, 1, tol=ref[2] * 1.2)
    assert a[:2] == b[:2] and a[0] == N.OK and a[1] < 400
    assert torch.equal(a[3], b[3])


def test_gives_up_and_recovers():
    import torch
    ref = _solve("qmt_jacobi_dirichlet", (64, 64, 64), 100, 0)
    N.call("qmt_set_wait_limit_ns", 1)
    try:
        st = _solve("qmt_jacobi_dirichlet", (64, 64, 64), 100, 0)
    finally:
        N.call("qmt_set_wait_limit_ns", 0)
    assert st[0] == N.CUDA_ERR and st[1] < 100
    again = _solve("qmt_jacobi_dirichlet", (64, 64, 64), 100, 0)
    assert again[:2] == (N.OK, 100) and torch.equal(again[3], ref[3])
