"""Factors whose rank is in the top eight of their limit where that limit, half of the basis rounded up to 16, is an
odd multiple of 8: the factor's columns rounded up to 16 then exceed the limit.

The density matrices are products of small whole numbers, exact in float32, so that the rank is what it is."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _molecule(basis, zs, rank, seed):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(len(zs) ** (1 / 3)))
    pos = np.array([(x, y, z) for x in range(k) for y in range(k) for z in range(k)][:len(zs)]) * 1.3
    rows = [[int(z), *(float(v) for v in p)] for z, p in zip(zs, pos + rng.uniform(-0.1, 0.1, pos.shape))]
    n = sum(sum(2 * L + 1 for L, _, _ in basis.shells64[z]) for z in zs)
    a = rng.integers(-3, 4, (n, rank)).astype(np.float64)
    assert np.linalg.matrix_rank(a) == rank
    return qmtools.Molecule(rows, a @ a.T, basis), n


# basis sizes 33, 70, 98, 294: limits 24, 40, 56, 152
@pytest.mark.parametrize("zs,prec", [([6, 6, 1], "fp16x3"), ([6] * 5, "fp16x3"), ([6] * 7, "fp16x3"),
                                     ([6] * 21, "fp16x3"), ([6, 6, 1], "bf16x3"), ([6] * 7, "bf16x3")])
def test_ranks_up_to_the_limit(basis, zs, prec):
    n = sum(sum(2 * L + 1 for L, _, _ in basis.shells64[z]) for z in zs)
    limit = (n + 15) // 16 * 8
    assert limit % 16 == 8
    for rank in range(limit - 8, limit + 1):
        mol, _ = _molecule(basis, zs, rank, rank)
        c = np.asarray(mol.coords).mean(axis=0)
        g = qmtools.Grid((1, 16, 16, 16), 0.5 / qmtools.ANG2BOR, list(c - 4.0 + 0.013))
        ref = qmtools.QMTools.Compute_density(g, mol, precision="fp64", rescale=False).qube.ravel()
        got = qmtools.QMTools.Compute_density(g, mol, precision=prec, rescale=False).qube.ravel()
        r = C.c_int()
        N.call("qmt_density_factor_rank", mol.handle, C.byref(r), N.stream_handle())
        assert r.value == rank
        # an FP32 addition per K-step, doubled by the square, and two operands of 2^-21 (fp16 pieces) or 2^-17
        tol = 2 * (n / 16 + 2) * 2.0 ** -23 + 4 * 2.0 ** (-21 if prec == "fp16x3" else -17)
        assert rel_l2(got, ref) <= tol
        mol.release()
