"""The factored density kernel at the edges of its units, ring and ranks, against the FP64 path.

Units of 16 columns: a molecule of one unit (padded to two), odd and even unit counts, light atoms that
leave a unit partly filled, shells that take the generic units; ranks at multiples of 16 and one past
them, where the factor stays in shared memory and where it streams, with two TMEM buffers
(rank <= 128) and one."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _molecule(basis, zs, rank, seed=0):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(len(zs) ** (1 / 3)))
    pos = np.array([(x, y, z) for x in range(k) for y in range(k) for z in range(k)][:len(zs)]) * 1.3
    pos = pos + rng.uniform(-0.1, 0.1, pos.shape)
    rows = [[int(z), *(float(v) for v in p)] for z, p in zip(zs, pos)]
    n = sum(sum(2 * L + 1 for L, _, _ in basis.shells64[z]) for z in zs)
    half = rng.standard_normal((n, rank)) / np.sqrt(n)
    return qmtools.Molecule(rows, half @ half.T, basis), n


def _grid(mol, n=16, step=0.5):
    c = np.asarray(mol.coords).mean(axis=0)
    return qmtools.Grid((1, n, n, n), step / qmtools.ANG2BOR, list(c - n * step / 2 + 0.013))


CASES = [
    ([1], 1), ([1, 1], 2), ([1, 1, 1, 1], 3),          # one or two units, light atoms
    ([6], 7), ([8, 1, 1], 5), ([6] * 3, 16), ([6] * 3 + [1] * 2, 17),
    ([35, 17, 17, 6, 1], 12),                          # generic units (Br, Cl)
    ([6] * 20, 64), ([6] * 21, 65),
    ([6] * 40, 128), ([6] * 41, 129), ([6] * 60, 250),  # streamed factor; one TMEM buffer past 128
]


@pytest.mark.parametrize("zs,rank", CASES, ids=[f"{len(z)}atoms-r{r}" for z, r in CASES])
def test_factored_matches_fp64(basis, zs, rank):
    mol, n = _molecule(basis, zs, rank)
    g = _grid(mol)
    ref = qmtools.QMTools.Compute_density(g, mol, precision="fp64", rescale=False).qube.ravel()
    got = qmtools.QMTools.Compute_density(g, mol, precision="fp16x3", rescale=False)
    r = C.c_int()
    N.call("qmt_density_factor_rank", mol.handle, C.byref(r), N.stream_handle())
    if rank <= (n + 15) // 16 * 8:
        assert r.value > 0      # the factored kernel ran (the float32 matrix may add small pivots)
    # per K-step one FP32 addition off by 2^-23 at most, doubled by the square; operands to 2^-21
    tol = 2 * (n / 16 + 2) * 2.0 ** -23 + 2 * 2.0 ** -21
    assert rel_l2(got.qube.ravel(), ref) <= tol
    mol.release()


@pytest.mark.parametrize("shape", [(13, 7, 5), (8, 4, 4), (1, 1, 1)])
def test_small_grids(basis, shape):
    """One tile, partial tiles and a single voxel: every voxel written once, nothing beyond."""
    import torch
    mol, n = _molecule(basis, [6, 1, 1, 1, 1], 5)
    nx, ny, nz = shape
    o = np.asarray(mol.coords).mean(axis=0) - np.array(shape) * 0.25
    out = {}
    for prec in ("fp64", "fp16x3"):
        q = torch.full((nx * ny * nz + 32,), -7.0, device="cuda")
        N.call("qmt_density", mol.handle, nx, ny, nz, 0.5, float(o[0]), float(o[1]), float(o[2]), 1, N.PREC[prec], 0,
               C.c_void_p(q.data_ptr()), None, N.stream_handle())
        out[prec] = q.cpu().numpy()
        assert np.all(out[prec][nx * ny * nz:] == -7.0)
    assert rel_l2(out["fp16x3"][:nx * ny * nz], out["fp64"][:nx * ny * nz]) <= 2e-6
    mol.release()
