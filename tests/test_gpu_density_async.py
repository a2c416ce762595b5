"""`qmt_density` without a host sum returns before the stream has done anything, the first call with a new density
matrix included, and gives what a call that waits gives."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N

pytestmark = pytest.mark.gpu

SHAPE = (40, 24, 32)


def _molecule(basis, zs):
    k = int(np.ceil(len(zs) ** (1 / 3)))
    pos = np.array([(x, y, z) for x in range(k) for y in range(k) for z in range(k)][:len(zs)]) * 1.4
    rows = [[int(z), *(float(v) for v in p)] for z, p in zip(zs, pos)]
    n = sum(sum(2 * L + 1 for L, _, _ in basis.shells64[z]) for z in zs)
    return qmtools.Molecule(rows, np.eye(n), basis), n


def _matrix(n, rank, seed, negative=False):
    rng = np.random.default_rng(seed)
    c = np.linalg.qr(rng.standard_normal((n, rank)))[0]
    w = np.ones(rank)
    if negative:
        w[-1] = -0.5
    return (c * w) @ c.T


def _density(mol, q, prec, sum_out=None):
    c = np.asarray(mol.coords).mean(axis=0) - np.array(SHAPE) * 0.2
    N.call("qmt_density", mol.handle, *SHAPE, 0.4, *(float(v) for v in c), 1, N.PREC[prec], 0, C.c_void_p(q.data_ptr()),
           C.byref(sum_out) if sum_out is not None else None, N.stream_handle())


# 20 carbon atoms: 280 functions, the fused kernel beside the factored one; 30: 420, the staged one
@pytest.mark.parametrize("prec", ["fp16x3", "bf16x3"])
@pytest.mark.parametrize("natoms,rank,negative", [(20, 60, False), (20, 16, False), (20, 200, False), (20, 60, True),
                                                  (30, 90, False), (30, 17, True)])
def test_first_call_with_a_matrix_does_not_wait(basis, natoms, rank, negative, prec):
    import torch
    N.ensure_device()
    mol, n = _molecule(basis, [6] * natoms)
    first, later, whole = (torch.empty(int(np.prod(SHAPE)), device="cuda") for _ in range(3))
    # (buffers and modules from a call with another matrix: growing a buffer may wait)
    for seed, r in ((1, 60), (2, n)):
        mol.set_dm(_matrix(n, r, seed))
        _density(mol, first, prec)
        torch.cuda.synchronize()
    mol.set_dm(_matrix(n, rank, 3, negative))
    torch.cuda.synchronize()
    ahead = torch.cuda.Event()
    torch.cuda._sleep(600_000_000)      # about 0.3 s
    ahead.record()
    _density(mol, first, prec)
    assert not ahead.query()
    _density(mol, later, prec)
    torch.cuda.synchronize()
    s = C.c_double()
    _density(mol, whole, prec, s)       # waits for the sum
    assert torch.equal(first, whole) and torch.equal(later, whole)
    _density(mol, later, prec)          # the host has seen the rank by now
    assert torch.equal(later, whole)
    mol.release()
