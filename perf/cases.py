"""The calls that programs make of this framework, as measurable cases.

Every case is one pass through the public entry points: the `QMTools` facade, `Molecule`,
`BatchEvaluator`, and the C ABI where a program keeps its results on the device (the facade's FFT
solve returns a host array).  Molecules are the synthetic ones of `qmtools.synthetic` (random
geometries of C, H, N, O at 1.8 bohr or more, cc-pVDZ).  Their density matrices are either `scf`
(the projector on the occupied orbitals, of rank sum Z / 2) or `corr` (every natural orbital
occupied a little, so of full rank, as a correlated calculation gives them).  The element lists
depend on the atom count alone, so a case's number of basis functions does not change with the seed.

`exact` evaluates the same inputs in FP64 with plain torch.
"""
import ctypes as C
import math
import struct
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "qmtools-pycuda_b200"))

import qmtools  # noqa: E402
from qmtools import _native as N  # noqa: E402
from qmtools import synthetic as syn  # noqa: E402
from qmtools.batch import BatchEvaluator  # noqa: E402

qmtools.set_verbose(False)

ANG2BOR = 1.8897259886
BOHR_ANG = 0.529177211
EPS0 = 0.0055263494
SIGMA, CUTOFF = 0.2, 6.0
F64 = torch.float64


def listed():
    return [
        # the smallest density call of the facade, host result included: launches and latency
        dict(name="density_c0_16", kind="density", natoms=8, side=6.0, nx=16, ny=16, nz=16, step=0.6, subgrid=1,
             precision="fp16x3", dm="scf", host=True),
        # the FP64 density of the small molecule on its own grid (first stage of its Jacobi route)
        dict(name="density_c0_64_fp64", kind="density", natoms=8, side=6.0, nx=64, ny=64, nz=64, step=0.2, subgrid=1,
             precision="fp64", dm="scf", host=False),
        # the headline step: density and free-space Hartree potential of the medium molecule
        dict(name="step_c1_128", kind="step", natoms=30, side=12.0, nx=128, ny=128, nz=128, step=0.15, padded=True),
        # one iteration of a self-consistent loop or one served request: a new density matrix each
        # call, density, potential returned to the host; a ragged grid
        dict(name="scf_20atoms", kind="scf", natoms=20, side=10.5, nx=88, ny=104, nz=96, step=0.17, padded=True),
        # the large molecule (N = 588) on its 192^3 grid
        dict(name="density_c2_192", kind="density", natoms=60, side=18.0, nx=192, ny=192, nz=192, step=0.12,
             subgrid=1, precision="fp16x3", dm="scf", host=False),
        # the largest served request: 120 atoms
        dict(name="density_120atoms", kind="density", natoms=120, side=19.0, nx=168, ny=168, nz=168, step=0.15,
             subgrid=1, precision="fp16x3", dm="scf", host=False),
        # a training molecule as the GA script prepares it: a correlated density matrix sampled on a
        # 2^3 subgrid, and its pseudo-field
        dict(name="train_fields", kind="train_fields", natoms=14, side=9.3, nx=56, ny=64, nz=48, step=0.3, iters=40),
        # one molecule's part of a GA element's fitness: automaton, rescale, difference
        dict(name="train_evaluate", kind="train_evaluate", natoms=14, side=9.3, nx=56, ny=64, nz=48, step=0.3,
             nlayers=4),
        # the Jacobi route of the small molecule: analytic boundary, 2000 sweeps
        dict(name="dirichlet_c0_64", kind="dirichlet", natoms=8, side=6.0, nx=64, ny=64, nz=64, step=0.2, sweeps=2000),
        # the same route of the medium molecule on its large grid: the boundary weighs as much as the sweeps
        dict(name="dirichlet_c1_128", kind="dirichlet", natoms=30, side=12.0, nx=128, ny=128, nz=128, step=0.15,
             sweeps=400),
        # the analytic potential on a whole grid
        dict(name="analytic_c0_64", kind="analytic", natoms=8, side=6.0, nx=64, ny=64, nz=64, step=0.2),
        # a batch of molecules of 5 to 60 atoms, densities and potentials in one graph launch
        dict(name="batch_16", kind="batch", count=16, lo=5, hi=60, step=0.15, pad=3.0, pick=3),
    ]


def draw(rng):
    """One more case of the listed kinds' ranges."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even8(lo, hi):
        return 8 * rng.randint(lo // 8, hi // 8)

    kind = rng.choice(["density", "density", "density", "step", "step", "scf", "batch", "train_fields",
                       "train_evaluate", "dirichlet", "dirichlet", "analytic"])
    if kind == "density":
        n = size(3, 120)
        while not _comparable(n):
            n = size(61, 120)
        side = round(syn.cube_side(n) * rng.uniform(1.0, 1.3), 2)
        sub = rng.choice([1, 1, 1, 2])
        prec = rng.choice(["fp16x3"] * 5 + ["fp32", "bf16x3", "tf32x3"])
        top = (80 if sub == 2 else 152) if n <= 60 else (56 if sub == 2 else 112)
        if prec in ("fp32", "tf32x3"):
            top = 56
        dm = rng.choice(["scf", "scf", "scf", "corr"])
        if dm == "corr" and n > 30:
            top = min(top, 72)
        nx, ny, nz = (even8(16, top) for _ in range(3))
        # the grid covers the molecule and up to 3 bohr a side
        step = round((side + rng.uniform(2.0, 6.0)) / max(nx, ny, nz), 4)
        return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz, step=step, subgrid=sub, precision=prec,
                    dm=dm, host=rng.random() < 0.3)
    if kind == "step":
        n = size(3, 60)
        side = round(syn.cube_side(n) * 1.05, 2)
        padded = rng.random() < 0.75
        # any length when padded; a periodic transform has the grid's own length (prime factors up to 127)
        nx, ny, nz = (rng.randint(20, 144) if padded else 2 * rng.randint(10, 72) for _ in range(3))
        return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz,
                    step=round((side + 6.0) / max(nx, ny, nz), 4), padded=padded)
    if kind == "scf":
        n = size(3, 60)
        side = round(syn.cube_side(n) * 1.05, 2)
        nx, ny, nz = (even8(32, 128) for _ in range(3))
        return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz,
                    step=round((side + 6.0) / max(nx, ny, nz), 4), padded=rng.random() < 0.75)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), lo=3, hi=60, step=round(rng.uniform(0.16, 0.3), 3), pad=3.0,
                    pick=rng.randint(0, 1 << 20))
    if kind == "train_fields":
        n = size(5, 20)
        side = round(syn.cube_side(n) * 1.05, 2)
        nx, ny, nz = (even8(32, 72) for _ in range(3))
        return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz,
                    step=round((side + 5.0) / min(nx, ny, nz), 4), iters=rng.randint(10, 60))
    if kind == "train_evaluate":
        n = size(5, 20)
        return dict(kind=kind, natoms=n, side=round(syn.cube_side(n) * 1.05, 2), nx=even8(32, 96), ny=even8(32, 96),
                    nz=even8(32, 96), step=round(rng.uniform(0.25, 0.4), 3), nlayers=rng.randint(1, 6))
    if kind == "dirichlet":
        n = size(3, 30)
        side = round(syn.cube_side(n) * 1.02, 2)
        nx, ny, nz = (even8(48, 128) for _ in range(3))
        return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz,
                    step=round(min(0.3, (side + 5.0) / min(nx, ny, nz)), 4), sweeps=2 * rng.randint(50, 500))
    n = size(3, 10)
    side = round(syn.cube_side(n), 2)
    nx, ny, nz = (even8(16, 72) for _ in range(3))
    return dict(kind=kind, natoms=n, side=side, nx=nx, ny=ny, nz=nz, step=round((side + 5.0) / max(nx, ny, nz), 4))


# ---- inputs ---------------------------------------------------------------------------------


class _Basis:
    """Shells of the cc-pVDZ file: per element [(L, exponents, coefficients)], as FP32 tables hold them."""

    def __init__(self, path):
        data = Path(path).read_bytes()
        self.shells, off = {}, 4
        for _ in range(struct.unpack_from("<i", data, 0)[0]):
            z, ns = struct.unpack_from("<ii", data, off)
            off += 8
            self.shells[z] = []
            for _ in range(ns):
                L, nc = struct.unpack_from("<ii", data, off)
                ac = np.frombuffer(data, "<f8", 2 * nc, off + 8).astype(np.float32).astype(np.float64)
                off += 8 + 16 * nc
                self.shells[z].append((L, ac[:nc], ac[nc:]))


_basis = _Basis(qmtools.BASIS_CCPVDZ)
_api_basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)

# real solid harmonics times r^l of the basis functions: L -> functions -> [(factor, powers of x, y, z)]
_S, _P, _D1, _D0, _D2 = 0.28209479177387814, 0.4886025119029199, 1.0925484305920792, 0.31539156525252005, 0.5462742152960396
_CART = {0: [[(_S, (0, 0, 0))]],
         1: [[(_P, (0, 0, 1))], [(_P, (1, 0, 0))], [(_P, (0, 1, 0))]],
         2: [[(2 * _D0, (0, 0, 2)), (-_D0, (2, 0, 0)), (-_D0, (0, 2, 0))], [(_D1, (1, 0, 1))], [(_D1, (0, 1, 1))],
             [(_D2, (2, 0, 0)), (-_D2, (0, 2, 0))], [(_D1, (1, 1, 0))]]}


def _types(natoms, side):
    return syn.element_list(natoms, np.random.default_rng(natoms), c0=natoms == 8 and side == 6.0)


def _shells(types):
    """[(atom, L, exponents, coefficients, first function)] and the number of functions."""
    out, f = [], 0
    for a, z in enumerate(types):
        for L, al, co in _basis.shells[int(z)]:
            out.append((a, L, al, co, f))
            f += 2 * L + 1
    return out, f


def _nbasis(types):
    return _shells(types)[1]


def _comparable(natoms):
    """False for the basis sizes whose unfactored tensor-core contraction had wrong results when these
    cases were first measured (its output panels were not a multiple of 32 columns wide, and the last
    16 of each were left out): there is nothing to compare other results of these sizes with."""
    k = -(-_nbasis(_types(natoms, 0.0)) // 64) * 64
    panels = -(-k // 256)
    return -(-k // panels // 16) * 16 % 32 == 0 or k <= 256


def _terms(coords, types):
    """Cartesian primitives: centre (n, 3), exponent, powers (n, 3), and their coefficients (n, N)."""
    shells, nf = _shells(types)
    atom, alpha, power, func, coef = [], [], [], [], []
    for a, L, al, co, f in shells:
        for x, c in zip(al, co):
            for k, terms in enumerate(_CART[L]):
                for w, e in terms:
                    atom.append(a)
                    alpha.append(x)
                    power.append(e)
                    func.append(f + k)
                    coef.append(w * c)
    m = torch.zeros(len(atom), nf, dtype=F64, device="cuda")
    m[torch.arange(len(atom)), torch.tensor(func)] = torch.tensor(coef, dtype=F64, device="cuda")
    return coords[atom], torch.tensor(alpha, dtype=F64, device="cuda"), torch.tensor(power, device="cuda"), m


def _overlap(coords, types):
    c, al, pw, m = _terms(coords, types)
    p = al[:, None] + al[None, :]
    s = torch.full_like(p, 1.0)
    for d in range(3):
        diff = c[:, None, d] - c[None, :, d]
        pa, pb, h = -al[None, :] / p * diff, al[:, None] / p * diff, 0.5 / p
        s11 = pa * pb + h
        s20, s02 = pa * pa + h, pb * pb + h
        s21, s12 = pa * s11 + h * (pa + pb), pb * s11 + h * (pa + pb)
        s22 = pa * s12 + h * (s02 + 2 * s11)
        table = [torch.ones_like(p), pb, s02, pa, s11, s12, s20, s21, s22]
        idx = 3 * pw[:, None, d] + pw[None, :, d]
        v = torch.zeros_like(p)
        for k, t in enumerate(table):
            v = torch.where(idx == k, t, v)
        s = s * v * torch.exp(-al[:, None] * al[None, :] / p * diff * diff) * torch.sqrt(math.pi / p)
    return m.T @ s @ m


def _matrix(coords, types, dm, seed):
    """Spin-up density matrix: C C^T over the occupied orbitals, C = S^-1/2 Q with Q random
    orthogonal, or over all of them with small natural occupations above the occupied ones."""
    n = _nbasis(types)
    w, u = torch.linalg.eigh(_overlap(coords, types))
    half = (u / torch.sqrt(torch.clamp(w, min=1e-8))) @ u.T
    g = torch.from_numpy(np.random.default_rng(seed).standard_normal((n, n))).cuda()
    q, r = torch.linalg.qr(g)
    c = half @ (q * torch.sign(torch.diagonal(r)))
    nocc = int(sum(types)) // 2
    if dm == "scf":
        c = c[:, :nocc]
        p = c @ c.T
    else:
        k = torch.arange(n, dtype=F64, device="cuda")
        occ = torch.where(k < nocc, 0.985 - 0.01 * k / max(nocc, 1), 0.02 * torch.exp(-6.0 * (k - nocc) / max(n - nocc, 1)))
        p = (c * occ) @ c.T
    return p.cpu().numpy().astype(np.float32)


def _geometry(natoms, side, shape, step, seed):
    """Atoms as the API takes them (rows Z, x, y, z in Angstrom), their FP32 bohr coordinates, and the
    grid's origin: the cube's centre at the grid's centre."""
    types = _types(natoms, side)
    xyz = syn.random_geometry(natoms, side, np.random.default_rng(seed))
    rows = [[int(z), *(float(v) for v in p / ANG2BOR)] for z, p in zip(types, xyz)]
    coords = (np.array(rows)[:, 1:] * ANG2BOR).astype(np.float32)
    origin = [float(np.float32(side / 2 - n * step / 2)) for n in shape]
    return types, rows, coords, origin


def _inputs(case, seed, dm="scf"):
    shape = (case["nx"], case["ny"], case["nz"])
    types, rows, coords, origin = _geometry(case["natoms"], case["side"], shape, case["step"], seed)
    c64 = torch.from_numpy(coords).to("cuda", F64)
    h = float(np.float32(case["step"] / ANG2BOR * ANG2BOR))
    return dict(shape=shape, types=types, rows=rows, coords=c64, origin=origin, h=h, step=case["step"],
                dm=_matrix(c64, types, dm, 1000 + seed) if dm else None)


def _molecule(i, dm=None):
    dm = i["dm"] if dm is None else dm
    if dm is None:   # the path does not read it
        dm = np.eye(_nbasis(i["types"]), dtype=np.float32)
    return qmtools.Molecule(i["rows"], dm, _api_basis)


def _grid(i, nfields=1):
    return qmtools.Grid((nfields,) + i["shape"], i["step"] / ANG2BOR, i["origin"])


def _batch_inputs(case, seed):
    """The batch's molecules: the sizes and grids come from `pick`, the geometries from the seed."""
    sizes = np.random.default_rng(case["pick"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
    out = []
    for k, n in enumerate(int(v) for v in sizes):
        side = syn.cube_side(n) * 1.02
        pts = 8 * math.ceil((side + 2 * case["pad"]) / case["step"] / 8)
        one = dict(natoms=n, side=side, nx=pts, ny=pts, nz=max(8, pts - 8 * (k % 3)), step=case["step"])
        out.append(_inputs(one, seed * 1000 + k))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        inp = _batch_inputs(case, seed)
        mols = [_molecule(i) for i in inp]
        return dict(kind=kind, ev=BatchEvaluator(mols, [_grid(i) for i in inp]))
    dm = {"density": case.get("dm"), "train_fields": "corr", "train_evaluate": None}.get(kind, "scf")
    i = _inputs(case, seed, dm)
    if kind == "scf":
        # the molecule as the loop holds it (an earlier matrix) and the matrix of this call
        first = _matrix(i["coords"], i["types"], "scf", 5000 + seed)
        mol = _molecule(i, first)
    else:
        mol = _molecule(i)
    s = dict(case, kind=kind, mol=mol, new_dm=i["dm"])
    nx, ny, nz = i["shape"]
    if kind == "step":
        mol.handle
        s.update(q=torch.empty(nx * ny * nz, device="cuda"), v=torch.empty(nx * ny * nz, device="cuda"),
                 geom=(nx, ny, nz, i["h"], *i["origin"]))
        return s
    s["grid"] = _grid(i)
    if kind == "dirichlet":
        s["grid"].field(0).copy_(_density(i).float())
    if kind == "train_evaluate":
        f, ref = _train_grids(i)
        s.update(field=torch.cat([torch.zeros_like(f), f]), out=_grid(i), ref=_grid(i))
        s["ref"].field(0).copy_(ref)
        g = np.random.default_rng(seed)
        s["params"] = ((2 * g.random(272 * case["nlayers"] + 29) - 1) * 0.3).astype(np.float32)
    return s


def _train_grids(i):
    """A pseudo-field and a reference density of the shape and range that training meets."""
    d = torch.stack([(_points(i) - c).norm(dim=1) for c in i["coords"]])
    z = torch.tensor(i["types"], dtype=F64, device="cuda")[:, None]
    ref = (z * torch.exp(-2.0 * d)).sum(0)
    return (0.2 * z * torch.exp(-d)).sum(0).float(), (ref * (float(z.sum()) / ref.sum())).float()


def run(s):
    kind, mol, T = s["kind"], s.get("mol"), qmtools.QMTools
    if kind == "density":
        g = T.Compute_density(s["grid"], mol, subgrid=s["subgrid"], precision=s["precision"], copyBack=s["host"])
        return g.qube if s["host"] else g.field(0)
    if kind == "step":
        q, v, st = C.c_void_p(s["q"].data_ptr()), C.c_void_p(s["v"].data_ptr()), N.stream_handle()
        N.call("qmt_density", mol.handle, *s["geom"], 1, N.PREC["fp16x3"], 1, q, None, st)
        N.call("qmt_fft_poisson", mol.handle, *s["geom"], SIGMA, CUTOFF, int(s["padded"]), q, v, st)
        return s["q"], s["v"]
    if kind == "scf":
        mol.set_dm(s["new_dm"])
        q = T.Compute_density(s["grid"], mol, copyBack=False)
        return q.field(0), T.Compute_hartree_fft(q, mol, sigma=SIGMA, cutoff=CUTOFF, padded=s["padded"])
    if kind == "batch":
        s["ev"].run()
        s["ev"].synchronize()
        return s["ev"].q, s["ev"].v
    if kind == "train_fields":
        q = T.Compute_density(s["grid"], mol, subgrid=2, copyBack=False)
        v = T.Compute_VNe(s["grid"], mol, adsorb=0.05, diff=0.02, tolerance=1e-12, maxiters=s["iters"], copyBack=False)
        return q.field(0), v.field(0)
    if kind == "train_evaluate":
        out, p = s["out"], s["params"]
        N.call("qmt_nn_singleshot", s["nx"], s["ny"], s["nz"], float(str(out.step)), C.c_void_p(s["field"].data_ptr()),
               C.c_void_p(out.field(0).data_ptr()), C.c_void_p(p.ctypes.data), int(p.size), s["nlayers"],
               N.stream_handle())
        T.Compute_qscale(out, mol.qtot / T.Compute_qtot(out))
        return out.field(0), T.Compute_qdiff(out, s["ref"])
    if kind == "dirichlet":
        return T.Compute_hartree_dirichlet(s["grid"], mol, max_sweeps=s["sweeps"], copyBack=False).field(0)
    T.Compute_hartree(s["grid"], mol, copyBack=False)
    return s["grid"].field(0)


# ---- what a pass cannot do without ----------------------------------------------------------


def _density_work(types, npts, sub, dm):
    n = _nbasis(types)
    rank = int(sum(types)) // 2 if dm == "scf" else n
    return 4 * npts + 4 * n * n, npts * sub ** 3 * 2.0 * rank * (n + 1)


def _fft_work(shape, padded):
    m = math.prod(shape) * (8 if padded else 1)
    return 8 * math.prod(shape), 2 * 2.5 * m * math.log2(m)


def _analytic_flops(types, npts):
    prims = sum(len(al) for _, _, al, _, _ in _shells(types)[0])
    return npts * (prims * (prims + 1) / 2) * 40.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        sizes = np.random.default_rng(case["pick"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
        for k, n in enumerate(int(v) for v in sizes):
            side = syn.cube_side(n) * 1.02
            pts = 8 * math.ceil((side + 2 * case["pad"]) / case["step"] / 8)
            shape = (pts, pts, max(8, pts - 8 * (k % 3)))
            d, p = _density_work(_types(n, side), math.prod(shape), 1, "scf"), _fft_work(shape, True)
            b, f = b + d[0] + 4 * math.prod(shape), f + d[1] + p[1]
        return dict(bytes=b, flops=f)
    types, shape = _types(case["natoms"], case["side"]), (case["nx"], case["ny"], case["nz"])
    npts = math.prod(shape)
    if kind == "density":
        b, f = _density_work(types, npts, case["subgrid"], case["dm"])
    elif kind in ("step", "scf"):
        (b, f), (_, f2) = _density_work(types, npts, 1, "scf"), _fft_work(shape, case["padded"])
        b, f = b + 4 * npts, f + f2
    elif kind == "train_fields":
        b, f = _density_work(types, npts, 2, "corr")
        b, f = b + 4 * npts, f + 2 * (case["iters"] + 1) * 56.0 * npts
    elif kind == "train_evaluate":
        b, f = 12 * npts, npts * 26 * (2.0 * 272 * case["nlayers"] + 36)
    elif kind == "dirichlet":
        shell = npts - math.prod(n - 2 for n in shape)
        b, f = 8 * npts, 8.0 * npts * case["sweeps"] + _analytic_flops(types, shell)
    else:
        b, f = 4 * npts, _analytic_flops(types, npts)
    return dict(bytes=b, flops=f)


# ---- the same results in FP64 ---------------------------------------------------------------


def _points(i, offset=(0.5, 0.5, 0.5)):
    """Positions origin + (index + offset) h of the grid, x fastest."""
    x, y, z = ((torch.arange(n, dtype=F64, device="cuda") + o) * i["h"] + p
               for n, o, p in zip(i["shape"], offset, i["origin"]))
    z, y, x = torch.meshgrid(z, y, x, indexing="ij")
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)], dim=1)


def _phi(pts, coords, types):
    out = torch.empty(pts.shape[0], _nbasis(types), dtype=F64, device="cuda")
    at = None
    for a, L, al, co, f in _shells(types)[0]:
        if a != at:
            at, d = a, pts - coords[a]
            r2 = (d * d).sum(1)
            x, y, z = d.unbind(1)
        rad = torch.zeros_like(r2)
        for e, c in zip(al, co):
            rad += float(c) * torch.exp(-float(e) * r2)
        if L == 0:
            out[:, f] = _S * rad
        elif L == 1:
            for k, v in enumerate((z, x, y)):
                out[:, f + k] = _P * v * rad
        else:
            for k, v in enumerate((_D0 * (2 * z * z - x * x - y * y), _D1 * x * z, _D1 * z * y, _D2 * (x * x - y * y),
                                   _D1 * x * y)):
                out[:, f + k] = v * rad
    return out


def _density(i, sub=1, scale=True):
    """Electrons per voxel, scaled to the nuclear charge."""
    p = torch.from_numpy(i["dm"]).to("cuda", F64)
    p = torch.tril(p) + torch.tril(p, -1).T
    q = 0.0
    offs = [(k + 0.5) / sub for k in range(sub)]
    chunk = max(4096, (1 << 27) // p.shape[0])
    for ox in offs:
        for oy in offs:
            for oz in offs:
                parts = []
                for pts in _points(i, (ox, oy, oz)).split(chunk):
                    phi = _phi(pts, i["coords"], i["types"])
                    parts.append(((phi @ p) * phi).sum(1))
                q = q + torch.cat(parts)
    q = q * (2.0 * i["h"] ** 3 / sub ** 3)
    return q * (float(sum(i["types"])) / q.sum()) if scale else q


def _poisson(i, q, padded):
    """Potential in volts, (nx, ny, nz), of the electrons and Gaussian nuclei."""
    nx, ny, nz = i["shape"]
    h = i["h"] / ANG2BOR
    rho = -q.reshape(nz, ny, nx).permute(2, 1, 0) / h ** 3
    ax = [o / ANG2BOR + (torch.arange(n, dtype=F64, device="cuda") + 0.5) * h for n, o in zip(i["shape"], i["origin"])]
    norm = 1.0 / (SIGMA ** 3 * (2 * math.pi) ** 1.5)
    for c, z in zip(i["coords"] * BOHR_ANG, i["types"]):
        r2 = ((ax[0] - c[0]) ** 2)[:, None, None] + ((ax[1] - c[1]) ** 2)[None, :, None] + ((ax[2] - c[2]) ** 2)[None, None, :]
        rho = rho + torch.where(r2 <= (CUTOFF * SIGMA) ** 2, float(z) * norm * torch.exp(-r2 / (2 * SIGMA ** 2)), 0.0)
    if not padded:
        k = [torch.fft.fftfreq(n, d=h, dtype=F64, device="cuda") for n in (nx, ny, nz)]
        k2 = (k[0] ** 2)[:, None, None] + (k[1] ** 2)[None, :, None] + (k[2] ** 2)[None, None, :]
        k2[0, 0, 0] = 1.0
        f = torch.fft.fftn(rho / EPS0) / (4 * math.pi ** 2 * k2)
        f[0, 0, 0] = 0.0
        return torch.fft.ifftn(f).real
    m = (2 * nx, 2 * ny, 2 * nz)
    a = [torch.arange(n, dtype=F64, device="cuda") for n in m]
    a = [torch.minimum(v, n - v) * h for v, n in zip(a, m)]
    r = torch.sqrt((a[0] ** 2)[:, None, None] + (a[1] ** 2)[None, :, None] + (a[2] ** 2)[None, None, :])
    g = torch.where(r > 0, 1.0 / r, 2.3800772417 / h) / (4 * math.pi * EPS0)
    v = torch.fft.irfftn(torch.fft.rfftn(rho, s=m) * torch.fft.rfftn(g), s=m)
    return v[:nx, :ny, :nz] * h ** 3


def _hermite(la, lb, a, b, xa, xb):
    """E[t] for t <= la + lb of a Gaussian product in one direction, over tensors of pairs."""
    p = a + b
    pa, pb, half = b / p * (xb - xa), a / p * (xa - xb), 0.5 / p
    e = [torch.ones_like(p)]
    for x in [pa] * la + [pb] * lb:
        e = [(x * e[t] if t < len(e) else 0.0) + (half * e[t - 1] if t else 0.0)
             + ((t + 1) * e[t + 1] if t + 1 < len(e) else 0.0) for t in range(len(e) + 1)]
    return e


def _potential(i, pts):
    """Analytic potential of the molecule's electrons and nuclei at the points (a.u.): the products of
    primitive shells in Hermite Gaussians, their potentials by the Boys-function recursion."""
    p = torch.from_numpy(i["dm"]).to("cuda", F64)
    p = torch.tril(p) + torch.tril(p, -1).T
    prims = {0: [], 1: [], 2: []}
    for a, L, al, co, f in _shells(i["types"])[0]:
        prims[L] += [(a, float(x), float(c), f) for x, c in zip(al, co)]
    v = torch.zeros(pts.shape[0], dtype=F64, device="cuda")
    for c, z in zip(i["coords"], i["types"]):
        v += float(z) / (pts - c).norm(dim=1)
    for la in range(3):
        for lb in range(la, 3):
            na, nb = len(prims[la]), len(prims[lb])
            if not na or not nb:
                continue
            ia, ib = (t.reshape(-1) for t in torch.meshgrid(torch.arange(na), torch.arange(nb), indexing="ij"))
            if la == lb:
                keep = ia <= ib
                ia, ib = ia[keep], ib[keep]
            fac = torch.where((ia == ib) & (la == lb), 1.0, 2.0).to("cuda", F64)
            A, B = (torch.tensor(prims[L], dtype=F64, device="cuda")[k.cuda()] for L, k in ((la, ia), (lb, ib)))
            ra, rb = i["coords"][A[:, 0].long()], i["coords"][B[:, 0].long()]
            a, b = A[:, 1], B[:, 1]
            s = a + b
            k = fac * A[:, 2] * B[:, 2] * torch.exp(-a * b / s * ((ra - rb) ** 2).sum(1)) * 2 * math.pi / s
            e = {(x, y, d): _hermite(x, y, a, b, ra[:, d], rb[:, d])
                 for x in range(la + 1) for y in range(lb + 1) for d in range(3)}
            coef = {}
            for u, ta in enumerate(_CART[la]):
                for w, tb in enumerate(_CART[lb]):
                    weight = k * p[A[:, 3].long() + u, B[:, 3].long() + w]
                    for ca, pa in ta:
                        for cb, pb in tb:
                            ex, ey, ez = (e[(pa[d], pb[d], d)] for d in range(3))
                            for t, vx in enumerate(ex):
                                for m, vy in enumerate(ey):
                                    for n, vz in enumerate(ez):
                                        coef[(t, m, n)] = coef.get((t, m, n), 0.0) + ca * cb * weight * vx * vy * vz
            size = sum(c.abs() for c in coef.values())
            live = size > 1e-18 * size.max()
            _add_pairs(v, pts, la + lb, s[live], ((a[:, None] * ra + b[:, None] * rb) / s[:, None])[live],
                       {q: c[live] for q, c in coef.items()})
    return v


def _add_pairs(v, pts, lmax, s, centre, coef):
    """v -= 2 sum over pairs and Hermite orders of coef R_tuv(s, centre - point)."""
    np_, chunk = pts.shape[0], max(1, (1 << 24) // pts.shape[0])
    for at in range(0, s.shape[0], chunk):
        sl = slice(at, at + chunk)
        x, y, z = (centre[sl, d, None] - pts[None, :, d] for d in range(3))
        q = s[sl, None]
        t = torch.clamp(q * (x * x + y * y + z * z), min=1e-12)
        nu = torch.tensor(lmax + 0.5, dtype=F64, device="cuda")
        f = torch.special.gammainc(nu, t) * math.gamma(lmax + 0.5) / (2 * t ** (lmax + 0.5))
        boys, et = [f], torch.exp(-t)
        for n in range(lmax - 1, -1, -1):
            f = (2 * t * f + et) / (2 * n + 1)
            boys.insert(0, f)
        table = {(n, 0, 0, 0): (-2 * q) ** n * boys[n] for n in range(lmax + 1)}

        def r(n, i, j, k):
            key = (n, i, j, k)
            if key not in table:
                if i:
                    val = x * r(n + 1, i - 1, j, k) + ((i - 1) * r(n + 1, i - 2, j, k) if i > 1 else 0.0)
                elif j:
                    val = y * r(n + 1, i, j - 1, k) + ((j - 1) * r(n + 1, i, j - 2, k) if j > 1 else 0.0)
                else:
                    val = z * r(n + 1, i, j, k - 1) + ((k - 1) * r(n + 1, i, j, k - 2) if k > 1 else 0.0)
                table[key] = val
            return table[key]

        acc = torch.zeros(x.shape, dtype=F64, device="cuda")
        for (i, j, k), c in coef.items():
            acc += c[sl, None] * r(0, i, j, k)
        v -= 2.0 * acc.sum(0)


def _seed_charges(i):
    """Each nucleus on the eight nodes around it, as the seed kernel weighs them."""
    nx, ny, nz = i["shape"]
    q = torch.zeros(nz, ny, nx, dtype=F64, device="cuda")
    for c, z in zip(i["coords"].cpu().numpy().astype(np.float32), i["types"]):
        rel = (c - np.array(i["origin"], dtype=np.float32)).astype(np.float64)
        base = np.floor(rel.astype(np.float32) / np.float32(i["h"])).astype(int)
        for t in np.ndindex(2, 2, 2):
            k = base + t
            q[k[2], k[1], k[0]] = float(z) * float(np.prod(np.abs(rel - k * i["h"]) / i["h"]))
    return q


def _relax(i, q, sweeps):
    nx, ny, nz = i["shape"]
    rho = (_seed_charges(i) - q.float().to(F64).reshape(nz, ny, nx)) / i["h"] ** 3
    pts = _points(i).reshape(nz, ny, nx, 3)
    shell = torch.ones(nz, ny, nx, dtype=torch.bool, device="cuda")
    shell[1:-1, 1:-1, 1:-1] = False
    v = torch.zeros(nz, ny, nx, dtype=F64, device="cuda")
    v[shell] = _potential(i, pts[shell])
    f = (4 * math.pi * i["h"] ** 2) * rho[1:-1, 1:-1, 1:-1]
    for _ in range(sweeps):
        s = (v[1:-1, 1:-1, :-2] + v[1:-1, 1:-1, 2:] + v[1:-1, :-2, 1:-1] + v[1:-1, 2:, 1:-1]
             + v[:-2, 1:-1, 1:-1] + v[2:, 1:-1, 1:-1] + f) / 6.0
        v[1:-1, 1:-1, 1:-1] = s
    return v.reshape(-1)


def _neighbours():
    return [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1) if (x, y, z) != (0, 0, 0)]


def _pseudo_field(i, ads, dif, pairs):
    nx, ny, nz = i["shape"]
    src = torch.zeros(nx * ny * nz, dtype=F64, device="cuda")
    for c, z in zip(i["coords"], i["types"]):
        d = (_points(i) - c).norm(dim=1)
        src += torch.where(d < math.sqrt(3.0) * i["h"], float(z) * torch.exp(-d), 0.0)
    src = src.reshape(nz, ny, nx)
    v = torch.zeros_like(src)
    for _ in range(2 * pairs):
        w = (1.0 - dif * 16.794682450997072 - ads) * v + src
        for x, y, z in _neighbours():
            w += dif / math.sqrt(abs(x) + abs(y) + abs(z)) * torch.roll(v, (-z, -y, -x), (0, 1, 2))
        v = torch.zeros_like(w)
        v[1:-1, 1:-1, 1:-1] = w[1:-1, 1:-1, 1:-1]
    return v.reshape(-1)


def _automaton(i, field, params, nlayers):
    """charge(v) = field(v) * sum over neighbours of the perceptron's output squared / distance weight / step."""
    nx, ny, nz = i["shape"]
    w = torch.zeros(272 * nlayers + 31, dtype=F64, device="cuda")
    w[:params.size] = torch.from_numpy(params).to("cuda", F64)
    f = field.to(F64).reshape(nz, ny, nx)
    out = torch.zeros_like(f)
    gridstep = float(str(np.float32(i["step"] / ANG2BOR * ANG2BOR)))
    for x, y, z in _neighbours():
        act = torch.cat([torch.stack([f, torch.roll(f, (-z, -y, -x), (0, 1, 2))]).reshape(2, -1),
                         w[:14, None].expand(14, f.numel())])
        at = 14
        for _ in range(nlayers):
            m = w[at:at + 272].reshape(16, 17)
            act = torch.tanh(m[:, :16] @ act + m[:, 16:])
            at += 272
        t = w[at:at + 16] @ act + w[at + 16]
        out += (t * t).reshape(f.shape) / math.sqrt(abs(x) + abs(y) + abs(z)) / gridstep
    return (f * out * 0.05234482976098482).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        qs, vs = [], []
        for i in _batch_inputs(case, seed):
            q = _density(i)
            pad = torch.zeros(-q.numel() % 64, dtype=F64, device="cuda")   # slices start at multiples of 64
            qs += [q, pad]
            vs += [_poisson(i, q, True).reshape(-1), pad]
        return torch.cat(qs), torch.cat(vs)
    dm = {"density": case.get("dm"), "train_fields": "corr", "train_evaluate": None}.get(kind, "scf")
    i = _inputs(case, seed, dm)
    if kind == "density":
        q = _density(i, case["subgrid"])
        return q.reshape(1, *i["shape"]) if case["host"] else q
    if kind in ("step", "scf"):
        q = _density(i)
        v = _poisson(i, q, case["padded"])
        return q, v if kind == "scf" else v.reshape(-1)
    if kind == "train_fields":
        return _density(i, 2), _pseudo_field(i, 0.05, 0.02, case["iters"] + 1)
    if kind == "train_evaluate":
        f, ref = _train_grids(i)
        g = np.random.default_rng(seed)
        q = _automaton(i, f, ((2 * g.random(272 * case["nlayers"] + 29) - 1) * 0.3).astype(np.float32), case["nlayers"])
        q = q * (float(sum(i["types"])) / q.sum())
        return q, float((q - ref.to(F64)).abs().sum())
    if kind == "dirichlet":
        return _relax(i, _density(i), case["sweeps"])
    return _potential(i, _points(i, (0.0, 0.0, 0.0)))
