"""Densities whose matrix is factored because of the size of the grid: from 8192 tiles of 128 sample points on, any
positive semi-definite matrix of up to 256 functions."""
import ctypes as C

import numpy as np
import pytest

import qmtools
from qmtools import _native as N

pytestmark = pytest.mark.gpu

SMALL, LARGE = (24, 16, 16), (104, 104, 104)     # 48 and 8788 tiles


def _molecule(basis, zs, matrix, seed=0):
    """`matrix`(n, generator) -> the density matrix."""
    rng = np.random.default_rng(seed)
    k = int(np.ceil(len(zs) ** (1 / 3)))
    pos = np.array([(x, y, z) for x in range(k) for y in range(k) for z in range(k)][:len(zs)]) * 1.4
    rows = [[int(z), *(float(v) for v in p)] for z, p in zip(zs, pos + rng.uniform(-0.1, 0.1, pos.shape))]
    n = sum(sum(2 * L + 1 for L, _, _ in basis.shells64[z]) for z in zs)
    return qmtools.Molecule(rows, matrix(n, rng), basis)


def _low_rank(rank):
    def m(n, rng):
        c = np.linalg.qr(rng.standard_normal((n, rank)))[0]
        return c @ c.T
    return m


def _density(mol, shape, prec, subgrid=1, wait=True):
    import torch
    span = float(np.ptp(np.asarray(mol.coords), axis=0).max()) + 6.0
    h = span / max(shape)
    org = [float(o) for o in np.asarray(mol.coords).mean(axis=0) - np.array(shape) * h / 2]
    q = torch.empty(int(np.prod(shape)), device="cuda")
    s = C.c_double()
    N.ensure_device()
    N.call("qmt_density", mol.handle, *shape, h, *org, subgrid, N.PREC[prec], 0, C.c_void_p(q.data_ptr()),
           C.byref(s) if wait else None, N.stream_handle())
    return q


def test_equal_calls_give_equal_results(basis):
    """A molecule whose charge rules out a rank of half of N (nine bromine atoms: 157 electron pairs, 243 functions) with
    a matrix of low rank all the same: a small grid's result does not depend on a large one's call before it."""
    import torch
    mol = _molecule(basis, [35] * 9, _low_rank(40))
    before = _density(mol, SMALL, "fp16x3")
    _density(mol, LARGE, "fp16x3")
    assert torch.equal(_density(mol, SMALL, "fp16x3"), before)
    mol.release()


def _full_rank(n, rng):
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    return (q * np.where(np.arange(n) < n // 3, 0.98, 0.02)) @ q.T


def _rank(mol):
    r = C.c_int()
    N.call("qmt_density_factor_rank", mol.handle, C.byref(r), N.stream_handle())
    return r.value


def test_rank_of_the_last_call(basis):
    """The rank that is asked for is that of the last call's contraction, whatever has been factored."""
    mol = _molecule(basis, [6] * 6 + [1] * 4, _full_rank)
    n = int(mol.norbs)
    for shape, prec, path, rank in ((LARGE, "fp16x3", 0, n), (SMALL, "fp16x3", 0, 0), (LARGE, "fp16x3", 0, n),
                                    (LARGE, "fp16x3", 2, 0), (LARGE, "fp16x3", 0, n), (SMALL, "fp64", 0, 0)):
        N.call("qmt_set_density_path", path)
        try:
            _density(mol, shape, prec)
        finally:
            N.call("qmt_set_density_path", 0)
        assert _rank(mol) == rank, (shape, prec, path)
    mol.release()


@pytest.mark.parametrize("rank", [20, 60, 104])
def test_rank_of_an_asynchronous_call(basis, rank):
    """The same where the call left the decision to the device: 104 functions, whose half is 52, rounded up to 56."""
    mol = _molecule(basis, [6] * 6 + [1] * 4, _full_rank)
    for shape, most in ((SMALL, 56), (LARGE, 104)):
        mol.set_dm(_low_rank(rank)(int(mol.norbs), np.random.default_rng(7)))
        _density(mol, shape, "fp16x3", wait=False)
        # (an exact projector has eigenvalues 0, which the float32 matrix has to rounding: a few more pivots at most)
        assert rank <= _rank(mol) <= most if rank <= most else _rank(mol) == 0
    mol.release()


def _captured(mol, shape, prec):
    """The density of an asynchronous call captured in a graph and replayed."""
    import torch
    span = float(np.ptp(np.asarray(mol.coords), axis=0).max()) + 6.0
    h = span / max(shape)
    org = [float(o) for o in np.asarray(mol.coords).mean(axis=0) - np.array(shape) * h / 2]
    q = torch.zeros(int(np.prod(shape)), device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        N.call("qmt_density", mol.handle, *shape, h, *org, 1, N.PREC[prec], 0, C.c_void_p(q.data_ptr()), None,
               N.stream_handle())
    g.replay()
    torch.cuda.synchronize()
    return q


def test_a_small_grid_is_captured_after_a_large_one(basis):
    """The operands of every grid exist after the first call."""
    import torch
    mol = _molecule(basis, [6] * 6 + [1] * 4, _full_rank)
    _density(mol, LARGE, "fp16x3")
    q = _captured(mol, SMALL, "fp16x3")
    assert torch.equal(q, _density(mol, SMALL, "fp16x3"))
    mol.release()


def test_a_large_grid_is_captured_after_a_small_one(basis):
    import torch
    mol = _molecule(basis, [6] * 6 + [1] * 4, _full_rank)
    ref = _density(mol, LARGE, "fp64")          # (this also makes the buffers that the large grid needs)
    _density(mol, SMALL, "fp16x3")
    q = _captured(mol, LARGE, "fp16x3")
    # an FP32 addition per K-step, doubled by the square, and two operands of 2^-21
    tol = 2 * (int(mol.norbs) / 16 + 2) * 2.0 ** -23 + 4 * 2.0 ** -21
    assert ((q.double() - ref.double()).norm() / ref.double().norm()).item() <= tol
    mol.release()


def _indefinite(n, rng):
    q = np.linalg.qr(rng.standard_normal((n, n)))[0]
    return (q * np.where(np.arange(n) < n // 3, 0.98, np.where(np.arange(n) < n - 3, 0.02, -0.05))) @ q.T


# 15, 42, 104, 148 and 256 functions, and 270, above the limit
FULL = [[1] * 3, [6] * 3, [6] * 6 + [1] * 4, [35, 17, 17] + [6] * 5 + [1] * 3, [6] * 17 + [17] * 1, [6] * 18 + [17]]


@pytest.mark.parametrize("zs", FULL, ids=[str(len(z)) for z in FULL])
@pytest.mark.parametrize("matrix", [_full_rank, _indefinite], ids=["definite", "indefinite"])
def test_full_rank_matrices_on_large_grids(basis, zs, matrix):
    """Against the FP64 path, on a 2^3 subgrid as training takes it and on single points, with the same molecule on a
    small grid before and after."""
    import torch
    mol = _molecule(basis, zs, matrix)
    n = int(mol.norbs)
    # an FP32 addition per K-step, doubled by the square of the factored contraction, or the row products' partial sums;
    # operands of 2^-21 each.  An indefinite matrix's terms cancel: as much again.
    tol = (2 * (n / 16 + 2) * 2.0 ** -23 + 4 * 2.0 ** -21) * (2 if matrix is _indefinite else 1)

    def off(a, b):
        return ((a.double() - b.double()).norm() / b.double().norm()).item()

    small = _density(mol, SMALL, "fp16x3")
    assert _rank(mol) == 0
    assert off(small, _density(mol, SMALL, "fp64")) <= tol
    for shape, sub in ((LARGE, 1), ((56, 48, 56), 2)):
        ref = _density(mol, shape, "fp64", sub)
        got = _density(mol, shape, "fp16x3", sub)
        assert _rank(mol) == (n if n <= 256 and matrix is _full_rank else 0)
        assert off(got, ref) <= tol
    assert torch.equal(_density(mol, SMALL, "fp16x3"), small)
    mol.release()


def test_full_rank_matrix_in_a_batch(basis, tmp_path):
    """One factored launch of a full-rank and a low-rank molecule, the full-rank one on a grid where it pays."""
    from qmtools.autotune import Tuner
    from qmtools.batch import BatchEvaluator
    mols = [_molecule(basis, [6] * 6 + [1] * 4, _full_rank), _molecule(basis, [6] * 6, _low_rank(17)),
            _molecule(basis, [6] * 6 + [1] * 4, _full_rank, 1)]
    shapes = [LARGE, (24, 32, 16), SMALL]
    grids = []
    for m, shape in zip(mols, shapes):
        c = np.asarray(m.coords)
        h = (float(np.ptp(c, axis=0).max()) + 6.0) / max(shape)
        grids.append(qmtools.Grid((1,) + shape, h / qmtools.ANG2BOR, list(c.mean(axis=0) - np.array(shape) * h / 2)))
    ev = BatchEvaluator(mols, grids, tuner=Tuner(path=tmp_path / "t.json", measure=False), hartree=False)
    try:
        assert ev.factored_count == 2
        ev.run()
        ev.synchronize()
        for k, (m, g) in enumerate(zip(mols, grids)):
            ref = qmtools.QMTools.Compute_density(g, m, precision="fp64").qube.ravel()
            tol = 2 * (int(m.norbs) / 16 + 2) * 2.0 ** -23 + 4 * 2.0 ** -21
            assert np.linalg.norm(ev.density(k).ravel() - ref) <= tol * np.linalg.norm(ref)
    finally:
        ev.close()
        for m in mols:
            m.release()
