"""Benchmark: density + Hartree grid points per second on the medium-molecule workload.

Workload (one step): a 30-atom molecule (C10 H14 N3 O3 drawn from a seed in a 12-bohr cube,
cc-pVDZ, N = 294 basis functions, closed-shell seeded density matrix) on a 128^3 grid at
0.15 bohr:
  1. electron density (tensor-core split contraction, default fp16x3), reference convention
     (electrons per voxel, rescaled to the nuclear charge);
  2. Hartree potential by the zero-padded (Hockney, free-space) FFT Poisson solve on a 256^3
     grid, nuclei as Gaussian charges (sigma 0.2 A), in FP32.
value = grid points (128^3 per step, summed over ranks) / second.  One process per GPU;
each rank evaluates its own copy of the workload (replicas, no collective on the path).

Timing: W warm-up steps, then K steps each bracketed by CUDA events on the launching
stream; before each timed step a 512 MiB buffer is written to flush L2.  Barrier and
synchronise on both sides; the reported time is the max over ranks.

`e2e` runs the same step through the public API starting from pinned host buffers
(coordinates and density matrix uploaded into the molecule handle, which re-derives its
device operands) and reads the potential grid back to the host every step.

Beside the headline step, rank 0 also reports (not part of `value`):
  * `plain_fp32`: the same step with the plain FP32 SIMT density path (the reference's
    precision), and the speed-up of the mixed-precision path over it;
  * `like_for_like`: the same density with the reference's own Poisson route (periodic FFT on
    the 128^3 grid itself), the step the `--impl reference` arm times;
  * `c0_route`: the small molecule (8 atoms, N = 58) on 64^3 at 0.2 bohr: FP64 density,
    analytic GTO potential on the outer shell, 2000 Dirichlet Jacobi sweeps, Hockney FFT on
    128^3;
  * `c2_sweep`: the large molecule (60 atoms, N = 588) on 192^3 at 0.12 bohr, the density in
    every precision, and an FP32 Jacobi solve to a relative FP64 residual of 1e-8;
  * `batched`: 64 molecules of 5-60 atoms (grids = bounding box + 3 bohr per side at
    0.15 bohr) in one CUDA graph (one persistent density launch for the factored molecules,
    autotuned paths for the others and FFT lengths), against the plain FP32 single-molecule path;
  * `serving`: Poisson request streams at 50, 200 and 800 req/s (atoms log-uniform 3-120)
    through the engine with p50/p99 latency, against serial plain FP32;
  * `cpu_baseline`: the FP64 NumPy/SciPy evaluation on a bounded sample;
  * `accuracy`: the mixed results scored against that FP64 evaluation (C1 density on sampled
    planes and Hartree on the full grid, every C2 variant on sampled planes).

`--impl reference` times the reference's own implementation of this path.  The reference is
GPU-only CUDA C driven from Python; its kernels, compiled from its sources into oracle/_ref,
run here with the reference facade's launch shapes and host steps (density kernel, grid
total and rescale, periodic cuFFT Poisson route), plus its analytic potential
(gpu_hartree_GTO) and Jacobi sweeps (gpu_hartree_iteration) on the small molecule's 64^3
grid.  Without those builds the FP64 CPU port of its algorithm is timed instead.

`--ncu-import CSV` turns an ncu metrics capture of the factored density kernel
(`--metrics dram__bytes_read.sum,dram__bytes_write.sum --csv`) into
profiles/density_factored_kernel_c1.traffic.json, which the bench reads for `roofline.traffic`.
"""
import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT / "qmtools-pycuda_b200"))
sys.path.insert(0, str(ROOT))

METRIC = "grid pts/s density+Hartree & req p50/p99, mixed vs plain FP32 at 1e-6 rel err"
UNIT = "grid_pts/s"
WORKLOAD = "medium molecule: 30 atoms C10H14N3O3, cc-pVDZ N=294, 128^3 grid @ 0.15 bohr, density + Hockney FFT Poisson on 256^3"


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return d.get("bf16_tflops", 1590.0), d.get("hbm_gbs", 6650.0), "measured"
    return 1590.0, 6650.0, "fallback"


class NvmlClockSampler:
    """SM clock and clock-event reasons polled through NVML every 10 ms in a thread."""

    def __init__(self, local):
        import pynvml
        import torch
        self.nv = pynvml
        pynvml.nvmlInit()
        uuid = "GPU-" + str(torch.cuda.get_device_properties(local).uuid)
        self.h = pynvml.nvmlDeviceGetHandleByUUID(uuid.encode() if isinstance(uuid, str) else uuid)
        self.max = float(pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM))
        self.samples = []
        self._stop = threading.Event()

    def _run(self):
        nv = self.nv
        get_reasons = getattr(nv, "nvmlDeviceGetCurrentClocksEventReasons",
                              getattr(nv, "nvmlDeviceGetCurrentClocksThrottleReasons", None))
        while not self._stop.is_set():
            try:
                self.samples.append((float(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM)),
                                     int(get_reasons(self.h)) if get_reasons else 0))
            except Exception:
                pass
            self._stop.wait(0.01)

    def __enter__(self):
        self.th = threading.Thread(target=self._run, daemon=True)
        self.th.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        self.th.join(timeout=2)

    def summary(self):
        nv = self.nv
        bits = {"hw_slowdown": "HwSlowdown", "hw_thermal_slowdown": "HwThermalSlowdown",
                "sw_thermal_slowdown": "SwThermalSlowdown", "sw_power_cap": "SwPowerCap"}
        reasons = set()
        for _, r in self.samples:
            for name, suffix in bits.items():
                b = getattr(nv, "nvmlClocksEventReason" + suffix, getattr(nv, "nvmlClocksThrottleReason" + suffix, 0))
                if r & b:
                    reasons.add(name)
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": self.max, "reasons": ["unsampled"], "samples": 0}
        return {"sm_mhz": float(np.median([c for c, _ in self.samples])), "sm_max_mhz": self.max,
                "reasons": sorted(reasons), "samples": len(self.samples), "source": "nvml 10 ms"}


def clock_sampler(local):
    try:
        return NvmlClockSampler(local)
    except Exception:
        return ClockSampler(local)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region (NVML fallback)."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        self.lines = []
        if self.proc is not None:
            self.proc.terminate()
            try:
                out, _ = self.proc.communicate(timeout=5)
            except Exception:
                self.proc.kill()
                out = ""
            self.lines = [l for l in out.splitlines() if l.strip()]

    def summary(self):
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in getattr(self, "lines", []):
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_setup(backend="nccl"):
    """One process per GPU (replicas): torchrun environment, short process-group timeout."""
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    pg = None
    if world > 1:
        import torch
        import torch.distributed as dist
        from datetime import timedelta
        if backend == "nccl":
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", timeout=timedelta(seconds=300),
                                    device_id=torch.device("cuda", local))
        else:
            dist.init_process_group(backend, timeout=timedelta(seconds=60))
        pg = dist
    return world, rank, local, pg


def _dev(pg):
    import torch
    return "cuda" if pg.get_backend() == "nccl" else "cpu"


def barrier(pg):
    if pg is not None:
        import torch
        pg.barrier()
        if _dev(pg) == "cuda":
            torch.cuda.synchronize()


def max_over_ranks(pg, v):
    """Timed regions are reported as the max over ranks."""
    if pg is None:
        return v
    import torch
    t = torch.tensor([v], dtype=torch.float64, device=_dev(pg))
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    return float(t.item())


def cpu_baseline_c1(sm, basis, qmtools, check=None):
    """FP64 NumPy/SciPy evaluation of the same step on a bounded sample, per grid point.

    Density: 4 z-planes (4*128^2 points) of the 128^3 grid through the oracle (chunked Phi,
    BLAS Phi@P, row-dot), extrapolated per point.  Hartree: one scipy.fft rfftn/irfftn
    Hockney convolution on the full 256^3 padded grid with all host cores.

    With `check` (host copies of device results) the same FP64 evaluation scores them; the
    scores are returned separately (accuracy, not timing): the C1 mixed density on the sampled
    planes and its Hockney potential on the full grid, and each C2 precision variant on its
    sampled planes.  Returns (baseline, accuracy or None).
    """
    import scipy.fft
    from oracle import density as od
    from oracle import poisson as op
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    nx, ny, nz, h, ox, oy, oz = g._geom()
    cores = os.cpu_count() or 1
    t0 = time.perf_counter()
    nzs = 4
    z0 = nz // 2
    q = od.density_qube_unscaled((nx, ny, nz), np.float32(h), (ox, oy, oz), mol.coords, mol.ALMOs, basis.alphas,
                                 basis.coeffs, mol.dm, zslab=(z0, z0 + nzs))
    t_dens = (time.perf_counter() - t0) / q.size
    M = 2 * nx
    rho = np.zeros((M, M, M))
    rho[:nx, :ny, :nz] = np.random.default_rng(0).random((nx, ny, nz))
    G = op.hockney_green((nx, ny, nz), h / op.ANG2BOR, (M, M, M))
    t1 = time.perf_counter()
    Gh = scipy.fft.rfftn(G, workers=cores)
    V = scipy.fft.irfftn(scipy.fft.rfftn(rho, workers=cores) * Gh, s=(M, M, M), workers=cores)
    t_fft = time.perf_counter() - t1
    npts = nx * ny * nz
    per_pt = t_dens + t_fft / npts
    out = {"value": 1.0 / per_pt, "unit": UNIT, "cores": cores, "kind": "port",
           "sample": f"density on {nzs} z-planes ({nzs * nx * ny} pts, FP64 NumPy, extrapolated per point) + "
                     f"one full {M}^3 scipy.fft Hockney convolution (workers={cores})",
           "density_s_per_pt": t_dens, "fft_s": t_fft}
    if check is None:
        return out, None
    acc = {"reference": "FP64 oracle (NumPy restatement of the reference algorithm) on the same inputs"}
    c1 = check["c1"]
    ref = np.asarray(q, dtype=np.float64).ravel()
    got = c1["q_raw"].reshape(nz, ny, nx)[z0:z0 + nzs].ravel().astype(np.float64)
    vref = op.hockney_poisson(c1["q"], (nx, ny, nz), h, (ox, oy, oz), mol.coords, mol.types, 0.2, 6)
    vref = np.asarray(vref, dtype=np.float64).ravel()
    vgot = c1["v"].astype(np.float64).ravel()
    acc["c1_mixed"] = {
        "precision": c1["precision"],
        "density_rel_l2": float(np.linalg.norm(got - ref) / np.linalg.norm(ref)),
        "density_max_abs": float(np.abs(got - ref).max()),
        "density_points": int(ref.size), "density_sample": f"z-planes {z0}..{z0 + nzs - 1} of {nz}",
        "hartree_rel_l2": float(np.linalg.norm(vgot - vref) / np.linalg.norm(vref)),
        "hartree_max_abs_volt": float(np.abs(vgot - vref).max()),
        "hartree_reference": "FP64 Hockney convolution (scipy) of the same density grid",
        "grid_electrons_fp64_path": c1["sum_fp64"], "grid_electrons_mixed": c1["sum_mixed"],
        "electron_count_2_trace_ps_fp64": c1["two_trace_ps"],
        "electron_count_error_mixed": abs(c1["sum_mixed"] - c1["two_trace_ps"]),
        "electron_count_error_fp64_path": abs(c1["sum_fp64"] - c1["two_trace_ps"])}
    if "c2" in check:
        c2 = check["c2"]
        m2 = c2["sm"].molecule(basis, qmtools.Molecule)
        gx, gy, gz, gh, gox, goy, goz = c2["geom"]
        refs = {z: np.asarray(od.density_qube_unscaled((gx, gy, gz), np.float32(gh), (gox, goy, goz), m2.coords,
                                                       m2.ALMOs, basis.alphas, basis.coeffs, m2.dm,
                                                       zslab=(z, z + 1)), dtype=np.float64).ravel()
                for z in c2["planes"]}
        r = np.concatenate([refs[z] for z in c2["planes"]])
        var = {}
        for prec, d in c2["variants"].items():
            gv = np.concatenate([d["planes"][z].astype(np.float64) for z in c2["planes"]])
            var[prec] = {"density_rel_l2": float(np.linalg.norm(gv - r) / np.linalg.norm(r)),
                         "density_max_abs": float(np.abs(gv - r).max()),
                         "grid_electrons": d["sum"],
                         "electron_count_error": abs(d["sum"] - c2["two_trace_ps"])}
        acc["c2_variants"] = {"sample": f"z-planes {list(c2['planes'])} of {gz} ({r.size} pts)",
                              "electron_count_2_trace_ps_fp64": c2["two_trace_ps"], "variants": var}
        m2.release()
    mol.release()
    return out, acc


def _requests(mols, basis, qmtools, serving, arrivals=None):
    out = []
    for i, m in enumerate(mols):
        out.append(serving.Request(m.molecule(basis, qmtools.Molecule), m.grid(qmtools.Grid),
                                   arrival=0.0 if arrivals is None else arrivals[i], rid=i))
    return out


def _engine_run(serving, reqs, slots, precision, realtime):
    import torch
    eng = serving.Engine(slots=slots, precision=precision)
    eng.warm(reqs)                              # steady state: every slot has served every request once
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    eng.run(reqs, realtime=realtime)
    torch.cuda.synchronize()
    wall = time.perf_counter() - t0
    eng.close()
    return wall


def batched(basis, qmtools, N, precision, reps=5):
    """The batch workload (64 molecules, 5-60 atoms, grids = bounding box + 3 bohr per side at
    0.15 bohr) through BatchEvaluator, all in one CUDA graph: one density launch for the factored
    molecules, the fused and staged paths for the rest, Hockney solves with tuned padding;
    against the plain FP32 single-molecule path (SIMT FP32 density + Hockney solve per molecule,
    handles built beforehand).  Device time with CUDA events.  Two graphs: `value` with every
    molecule's factored density matrix (factors built and checked when the batch is created,
    `setup_s`); `refresh` re-derives the unfactored operands inside the graph, so that new density
    matrices uploaded between replays are followed, and its end-to-end figure adds, per replay,
    the upload of every density matrix from pinned memory and the download of every potential."""
    import ctypes as C
    import torch
    from qmtools import synthetic as syn
    from qmtools.autotune import Tuner
    from qmtools.batch import BatchEvaluator
    bm = syn.batch_molecules(64)
    mols = [m.molecule(basis, qmtools.Molecule) for m in bm]
    grids = [m.grid(qmtools.Grid) for m in bm]
    pts = sum(int(g.npts) for g in grids)
    tuner = Tuner()

    def graph_ms(ev):
        ev.run()
        ev.synchronize()
        st = ev.stream
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        for _ in range(reps):
            ev.run()
        e1.record(st)
        e1.synchronize()
        return e0.elapsed_time(e1) / reps

    t0 = time.perf_counter()
    evf = BatchEvaluator(mols, grids, precision=precision, tuner=tuner, refresh=False)
    setup_f = time.perf_counter() - t0
    ms = graph_ms(evf)
    fact_info = {"fused_molecules": evf.fused_count, "factored_molecules": evf.factored_count,
                 "gpu_launches_per_batch": evf.launches_per_run, "setup_s": setup_f}
    evf.close()
    t0 = time.perf_counter()
    ev = BatchEvaluator(mols, grids, precision=precision, tuner=tuner, refresh=True)
    setup_s = time.perf_counter() - t0
    ms_ref = graph_ms(ev)
    st = ev.stream
    # end to end: density matrices up (pinned), graph, potentials down (pinned)
    dms = [torch.from_numpy(np.ascontiguousarray(m.dm, dtype=np.float32)).pin_memory() for m in mols]
    v_host = torch.empty(ev.v.numel(), dtype=torch.float32).pin_memory()
    sh = C.c_void_p(st.cuda_stream)

    def e2e():
        for m, d in zip(mols, dms):
            N.call("qmt_mol_set_dm", m.handle, C.c_void_p(d.data_ptr()), sh)
        ev.run()
        with torch.cuda.stream(st):
            v_host.copy_(ev.v, non_blocking=True)

    e2e()
    st.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(st)
    for _ in range(reps):
        e2e()
    e1.record(st)
    e1.synchronize()
    ms_e2e = e0.elapsed_time(e1) / reps
    ev.close()
    # plain FP32 single-molecule path, one molecule after another on the device
    cur = torch.cuda.current_stream()
    s0 = C.c_void_p(cur.cuda_stream)
    q = torch.empty(max(int(g.npts) for g in grids), device="cuda")
    v = torch.empty_like(q)

    def serial():
        for m, g in zip(mols, grids):
            nx, ny, nz, h, ox, oy, oz = g._geom()
            N.call("qmt_density", m.handle, nx, ny, nz, h, ox, oy, oz, 1, N.PREC["fp32"], 1,
                   C.c_void_p(q.data_ptr()), None, s0)
            N.call("qmt_fft_poisson", m.handle, nx, ny, nz, h, ox, oy, oz, 0.2, 6.0, 1, C.c_void_p(q.data_ptr()),
                   C.c_void_p(v.data_ptr()), s0)

    serial()
    torch.cuda.synchronize()
    ms32 = _events_ms(serial, 1)
    nfused = sum(1 for p in ev.paths if p == 2)
    for m in mols:
        m.release()
    return {"molecules": len(bm), "atoms": "uniform 5-60", "grid_pts": pts,
            "grids": "bounding box + 3 bohr per side at 0.15 bohr, multiples of 8",
            "value": pts / (ms / 1e3), "unit": UNIT, "ms_per_batch": ms,
            "factored": fact_info,
            "refresh": {"value": pts / (ms_ref / 1e3), "unit": UNIT, "ms_per_batch": ms_ref,
                        "speedup_vs_serial_plain_fp32": ms32 / ms_ref, "fused_molecules": ev.fused_count,
                        "gpu_launches_per_batch": ev.launches_per_run, "setup_s": setup_s},
            "e2e": {"value": pts / (ms_e2e / 1e3), "unit": UNIT, "ms_per_batch": ms_e2e,
                    "graph": "refresh (new density matrices uploaded every replay)",
                    "h2d_bytes": int(sum(d.numel() * 4 for d in dms)), "d2h_bytes": int(v_host.numel() * 4)},
            "serial_plain_fp32": {"value": pts / (ms32 / 1e3), "ms": ms32},
            "speedup_vs_serial_plain_fp32": ms32 / ms, "speedup_e2e_vs_serial_plain_fp32": ms32 / ms_e2e,
            "design": f"one CUDA graph per batch: persistent density launches over the tiles of "
                      f"{fact_info['fused_molecules']} molecules (factored density matrices), the staged "
                      f"path for the other {len(bm) - fact_info['fused_molecules']} "
                      f"({fact_info['factored_molecules']} of 64 factored in all), rescale, 64 Hockney "
                      f"solves with autotuned padding",
            "tuner": {"decisions_measured_now": tuner.measured, "cache": str(tuner.path),
                      "fused_chosen": nfused},
            "timing": "CUDA events around graph replays on the batch stream"}


def serving_streams(basis, qmtools, precision):
    """C4-like request streams through the continuous-batching engine."""
    from qmtools import serving
    from qmtools import synthetic as syn
    res = {}
    count = 32
    rates = (50.0, 200.0, 800.0)
    # the atom counts depend only on the seed, so every rate serves the same molecules
    mols = [m for _, m in syn.serving_stream(rates[0], count)]
    pts = sum(int(np.prod(m.grid_shape)) for m in mols)
    t_fp32 = _engine_run(serving, _requests(mols, basis, qmtools, serving), 1, "fp32", False)
    streams = {}
    for rate in rates:
        stream = syn.serving_stream(rate, count)
        arr = [t for t, _ in stream]
        reqs = _requests([m for _, m in stream], basis, qmtools, serving, arr)
        t_mix = _engine_run(serving, reqs, 8, precision, True)
        lat = serving.latency_stats(reqs)
        streams[f"{int(rate)}_req_s"] = {
            "rate_req_s": rate, "p50_ms": lat["p50_ms"], "p99_ms": lat["p99_ms"], "mean_ms": lat["mean_ms"],
            "value": pts / t_mix, "unit": UNIT, "makespan_s": t_mix, "arrival_span_s": arr[-1],
            "speedup_vs_serial_plain_fp32": t_fp32 / t_mix}
    res["serving"] = {"requests": count, "atoms": "log-uniform 3-120", "grid_pts": pts, "slots": 8,
                      "serial_plain_fp32": {"value": pts / t_fp32, "wall_s": t_fp32}, "streams": streams}
    return res


def _events_ms(fn, reps=1):
    """Mean duration of fn() over `reps` calls on the current stream, CUDA events."""
    import torch
    st = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(st)
    for _ in range(reps):
        fn()
    e1.record(st)
    e1.synchronize()
    return e0.elapsed_time(e1) / reps


def c0_route(basis, qmtools, N):
    """The small-molecule configuration end to end on the device: FP64 density on 64^3 at 0.2 bohr,
    the analytic GTO potential on the grid's outer shell, 2000 Dirichlet Jacobi sweeps (FP32,
    FP64 residual) and the Hockney FFT solve on 128^3; each stage timed with CUDA events."""
    import ctypes as C
    import torch
    from qmtools import synthetic as syn
    sm = syn.config_molecule("c0")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    nx, ny, nz, h, ox, oy, oz = g._geom()
    n = nx * ny * nz
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    q = torch.empty(n, device="cuda")
    seed = torch.zeros(n, device="cuda")
    rho = torch.empty(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    t = torch.empty(n, device="cuda")
    vfft = torch.empty(n, device="cuda")
    qs = C.c_double()
    sw, dl = C.c_int(), C.c_double()
    vp = lambda x: C.c_void_p(x.data_ptr())

    def density():
        N.call("qmt_density", mol.handle, nx, ny, nz, h, ox, oy, oz, 1, N.PREC["fp64"], 1, vp(q), None, st)

    def boundary():
        N.call("qmt_hartree_gto_boundary", mol.handle, nx, ny, nz, h, ox, oy, oz, vp(v), st)

    def jacobi():
        v.zero_()
        boundary()
        seed.zero_()
        N.call("qmt_density_seed", mol.handle, nx, ny, nz, h, ox, oy, oz, vp(seed), st)
        torch.sub(seed, q, out=rho)
        rho.mul_(1.0 / float(h) ** 3)
        N.call("qmt_jacobi_dirichlet", nx, ny, nz, h, vp(rho), vp(v), vp(t), 2000, 100, 0.0, C.byref(sw),
               C.byref(dl), st)

    def fft():
        N.call("qmt_fft_poisson", mol.handle, nx, ny, nz, h, ox, oy, oz, 0.2, 6.0, 1, vp(q), vp(vfft), st)

    for f in (density, boundary, jacobi, fft):
        f()
    torch.cuda.synchronize()
    ms = {"density_fp64": _events_ms(density, 3), "gto_boundary": _events_ms(boundary, 3),
          "jacobi_2000_sweeps_incl_boundary": _events_ms(jacobi, 1), "fft_hockney_128": _events_ms(fft, 5)}
    tot = ms["density_fp64"] + ms["jacobi_2000_sweeps_incl_boundary"] + ms["fft_hockney_128"]
    shell = n - (nx - 2) * (ny - 2) * (nz - 2)
    res = {"workload": f"C0: 8 atoms C2H6, N=58, 64^3 @ 0.2 bohr; FP64 density, GTO boundary ({shell} shell pts "
                       "at voxel centres), 2000 Dirichlet Jacobi sweeps FP32/FP64 residual, Hockney FFT 128^3",
           "ms": ms, "total_ms": tot, "value": n / (tot / 1e3), "unit": UNIT,
           "jacobi_sweeps": sw.value, "jacobi_fp64_residual": dl.value}
    mol.release()
    return res


def c2_sweep(basis, qmtools, N, planes=(48, 144)):
    """The large molecule (60 atoms, N = 588) on 192^3 at 0.12 bohr: the density in every
    precision (raw electrons per voxel, CUDA-event time per call), host copies of sampled
    z-planes for scoring against the FP64 oracle, and an FP32 Dirichlet Jacobi solve run until
    the FP64 residual sum |V_k - V_k-1| falls below 1e-8 of sum |V| (capped)."""
    import ctypes as C
    import torch
    from qmtools import synthetic as syn
    sm = syn.config_molecule("c2")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    nx, ny, nz, h, ox, oy, oz = g._geom()
    n = nx * ny * nz
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    q = torch.empty(n, device="cuda")
    vp = lambda x: C.c_void_p(x.data_ptr())
    tr = C.c_double()
    N.call("qmt_mol_trace_ps", mol.handle, C.byref(tr), st)
    out = {"workload": f"C2: 60 atoms C20H28N6O6, N={int(mol.norbs)}, 192^3 @ 0.12 bohr", "variants": {}}
    check = {"sm": sm, "geom": (nx, ny, nz, h, ox, oy, oz), "planes": planes, "variants": {},
             "two_trace_ps": 2.0 * tr.value}
    for prec in ("fp64", "fp32", "tf32", "tf32x3", "bf16", "bf16x3", "fp16x3"):
        s = C.c_double()

        def dens():
            N.call("qmt_density", mol.handle, nx, ny, nz, h, ox, oy, oz, 1, N.PREC[prec], 0, vp(q), None, st)

        dens()
        ms = _events_ms(dens, 1 if prec == "fp64" else 3)
        N.call("qmt_density", mol.handle, nx, ny, nz, h, ox, oy, oz, 1, N.PREC[prec], 0, vp(q), C.byref(s), st)
        qz = q.view(nz, ny, nx)
        check["variants"][prec] = {"planes": {z: qz[z].cpu().numpy().ravel().copy() for z in planes},
                                   "sum": s.value}
        out["variants"][prec] = {"ms": ms, "value": n / (ms / 1e3), "unit": UNIT, "grid_electrons": s.value}
    # Jacobi to a relative residual of 1e-8: charge = seed - fp16x3 density, boundary = GTO potential
    rho = torch.zeros(n, device="cuda")
    v = torch.zeros(n, device="cuda")
    t = torch.empty(n, device="cuda")
    N.call("qmt_density_seed", mol.handle, nx, ny, nz, h, ox, oy, oz, vp(rho), st)
    rho.sub_(q).mul_(1.0 / float(h) ** 3)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    N.call("qmt_hartree_gto_boundary", mol.handle, nx, ny, nz, h, ox, oy, oz, vp(v), st)
    e1.record()
    sweeps, rel, chunk, cap = 0, float("inf"), 5000, 100000
    jac_ms = 0.0
    sw, dl = C.c_int(), C.c_double()
    while sweeps < cap:
        ms = _events_ms(lambda: N.call("qmt_jacobi_dirichlet", nx, ny, nz, h, vp(rho), vp(v), vp(t), chunk, 100,
                                       0.0, C.byref(sw), C.byref(dl), st))
        jac_ms += ms
        sweeps += sw.value
        norm = float(v.double().abs().sum())
        rel = dl.value / norm
        if rel <= 1e-8:
            break
    out["jacobi_to_1e-8"] = {"sweeps": sweeps, "fp64_residual_sum_abs_dV": dl.value, "relative_residual": rel,
                             "converged": rel <= 1e-8, "cap_sweeps": cap, "ms": jac_ms,
                             "us_per_sweep": 1e3 * jac_ms / max(sweeps, 1),
                             "gto_boundary_ms": e0.elapsed_time(e1),
                             "residual": "FP64 sum |V_k - V_k-1| over the grid at the last sweep of a "
                                         f"{chunk}-sweep launch, relative to sum |V_k|"}
    mol.release()
    return out, check


def run_ours(args, world, rank, local, pg):
    import ctypes as C
    import torch
    import qmtools
    from qmtools import _native as N
    from qmtools import synthetic as syn
    qmtools.set_verbose(False)
    torch.cuda.set_device(local)
    basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)
    sm = syn.config_molecule("c1")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    if args.grid:
        # the same molecule on a smaller cube of the same spacing, centred on it (profiling cases)
        c = np.asarray(sm.coords_bohr).mean(axis=0)
        hb = sm.step_bohr
        g = qmtools.Grid((1, args.grid, args.grid, args.grid), hb / qmtools.ANG2BOR, list(c - args.grid * hb / 2))
    nx, ny, nz, h, ox, oy, oz = g._geom()
    npts = nx * ny * nz
    qgrid = qmtools.Grid.emptyAs(g)
    q = qgrid.tensor()
    vout = torch.empty(npts, dtype=torch.float32, device="cuda")
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")
    prec = N.PREC[args.precision]
    stream = torch.cuda.current_stream()
    sh = C.c_void_p(stream.cuda_stream)
    qsum = C.c_double()
    handle = mol.handle
    lib = N.load()

    def density(p=prec):
        N.call("qmt_density", handle, nx, ny, nz, h, ox, oy, oz, 1, p, 1, C.c_void_p(q.data_ptr()),
               C.byref(qsum), sh)

    def poisson(padded=1):
        N.call("qmt_fft_poisson", handle, nx, ny, nz, h, ox, oy, oz, 0.2, 6.0, padded, C.c_void_p(q.data_ptr()),
               C.c_void_p(vout.data_ptr()), sh)

    def step():
        density()
        poisson()

    def timed(fn, k, split=None):
        """Mean ms per step over k steps, CUDA events on the launching stream around each step, the
        L2 flushed before each; with `split` (density, rest) the density part is timed as well."""
        tot = 0.0
        dens = 0.0
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
        for _ in range(k):
            flush.fill_(1.0)
            ev[0].record(stream)
            if split is not None:
                split[0]()
                ev[1].record(stream)
                split[1]()
            else:
                fn()
                ev[1].record(stream)
            ev[2].record(stream)
            ev[2].synchronize()
            tot += ev[0].elapsed_time(ev[2])
            dens += ev[0].elapsed_time(ev[1])
        return tot / k, dens / k

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    barrier(pg)
    l0 = lib.qmt_launch_count()
    with clock_sampler(local) as clk:
        ms, dens_ms = timed(step, args.steps, split=(density, poisson))
    torch.cuda.synchronize()
    launches = lib.qmt_launch_count() - l0
    barrier(pg)
    ms = max_over_ranks(pg, ms)

    # end to end through the public API from pinned host buffers
    coords_h = torch.from_numpy(np.ascontiguousarray(mol.coords, dtype=np.float32)).pin_memory()
    dm_h = torch.from_numpy(np.ascontiguousarray(mol.dm, dtype=np.float32)).pin_memory()
    v_h = torch.empty(npts, dtype=torch.float32).pin_memory()

    def e2e_step(padded=1):
        N.call("qmt_mol_set_coords", handle, C.c_void_p(coords_h.data_ptr()), sh)
        N.call("qmt_mol_set_dm", handle, C.c_void_p(dm_h.data_ptr()), sh)
        density()
        poisson(padded)
        v_h.copy_(vout, non_blocking=True)

    for _ in range(max(1, args.warmup)):
        e2e_step()
    torch.cuda.synchronize()
    barrier(pg)
    e2e_ms, _ = timed(e2e_step, args.steps)
    e2e_ms = max_over_ranks(pg, e2e_ms)

    out = {
        "metric": METRIC, "value": world * npts / (ms / 1000.0), "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": args.precision,
        "data": "synthetic (seeded geometry and density matrix; no public dataset exists for this path)",
        "config": {"workload": WORKLOAD if not args.grid else WORKLOAD.replace("128^3", f"{args.grid}^3"),
                   "grid_pts_per_step": npts, "basis_functions": int(mol.norbs),
                   "density_precision": args.precision, "poisson": "Hockney free-space FFT, 256^3 padded, FP32",
                   "l2": "512 MiB flush written before every timed step", "parallelism": f"replicas x{world}"},
        "e2e": {"value": world * npts / (e2e_ms / 1000.0), "unit": UNIT,
                "h2d_bytes_per_step": int(coords_h.numel() * 4 + dm_h.numel() * 4),
                "d2h_bytes_per_step": int(v_h.numel() * 4)},
        "gpu_launches": int(launches),
        "gpu_launches_per_step": launches / args.steps,
        "gpu_launches_counted": "qmt_launch_count() difference around the timed steps (this library's kernels)",
        "clocks": clk.summary(),
    }
    # roofline of the dominant kernel: the density contraction, algorithmic flops npts(2N^2+2N)
    nb = int(mol.norbs)
    flops = npts * (2.0 * nb * nb + 2.0 * nb)
    peak_tf, hbm, kind = peaks()
    achieved = flops / (dens_ms / 1000.0) / 1e12
    traffic = profiled_traffic() if (args.precision == "fp16x3" and not args.grid) else None
    frank = C.c_int()
    N.call("qmt_density_factor_rank", handle, C.byref(frank), sh)
    frank = int(frank.value)
    r16 = max(16, (frank + 15) // 16 * 16)
    out["roofline"] = {"bound": "tensor",
                       "kernel": ("density_factored_kernel" if frank else "density_fused_kernel") +
                                 " (basis values in shared memory + tcgen05 contraction)",
                       "achieved": achieved, "peak": peak_tf, "unit": "TFLOP/s", "frac": achieved / peak_tf,
                       "peak_source": f"bf16_tflops burst, {kind}", "density_ms": dens_ms,
                       "algorithmic_flop_per_launch": flops,
                       "algorithmic_flop_definition": "npts (2 N^2 + 2 N): Phi P plus the row-dot",
                       "contraction": (f"factored density matrix P = L L^T, rank {frank}: rho = sum_k (Phi L)_k^2, "
                                       f"MMA N = {r16} x 3 products (large and small in two accumulators), "
                                       f"{npts * 2.0 * nb * r16 * 3:.3e} tensor flop per launch"
                                       if frank else "unfactored: Phi P (N columns) x 3 products, row-dot with Phi"),
                       "traffic": traffic["bytes_per_launch"] if traffic else None,
                       "traffic_unit": "DRAM bytes per launch (ncu, dram__bytes_read.sum + dram__bytes_write.sum)",
                       "traffic_source": traffic["source"] if traffic else None}
    # the basis evaluation's exponentials, counted separately (npts x primitives of all shells,
    # before screening): what bounds the SIMT half of the kernel
    almos = np.asarray(mol.ALMOs).reshape(-1, 4)
    shells = {(int(r[0]), int(r[3])) for r in almos}
    co = np.asarray(mol.basisset.coeffs)
    nprim = sum(int(np.count_nonzero(co[so:so + 20])) for _, so in shells)
    out["roofline"]["exponentials_per_launch"] = int(npts * nprim)
    out["roofline"]["exponentials_per_s"] = npts * nprim / (dens_ms / 1000.0)
    # the basis evaluation bounds the factored kernel: exponentials against the SFU rate (16 per
    # SM and clock, nominal, at the sampled clock)
    clk = out["clocks"].get("sm_mhz") or 1965.0
    sfu_peak = 16.0 * 148 * clk * 1e6
    out["roofline"]["sfu_exp_peak_per_s"] = sfu_peak
    out["roofline"]["sfu_frac"] = npts * nprim / (dens_ms / 1000.0) / sfu_peak
    check = None
    if world == 1 and not args.quick:
        # plain FP32 SIMT density (the reference's precision) on the same step
        def step32():
            density(N.PREC["fp32"])
            poisson()

        step32()
        ms32, _ = timed(step32, 5)
        out["plain_fp32"] = {"value": npts / (ms32 / 1000.0), "unit": UNIT, "ms_per_step": ms32,
                             "speedup_of_mixed": ms32 / ms}

        # the reference's own Poisson route (periodic, on the 128^3 grid itself): the step the
        # reference arm times
        def step_periodic():
            density()
            poisson(0)

        step_periodic()
        msp, _ = timed(step_periodic, args.steps)
        e2e_step(0)
        e2e_p, _ = timed(lambda: e2e_step(0), args.steps)
        out["like_for_like"] = {
            "workload": WORKLOAD.replace("density + Hockney FFT Poisson on 256^3",
                                         "density + periodic FFT Poisson on 128^3 (the reference's solve)"),
            "value": npts / (msp / 1e3), "unit": UNIT, "ms_per_step": msp,
            "e2e": {"value": npts / (e2e_p / 1e3), "unit": UNIT}}
        # device results scored against the FP64 oracle in the CPU leg
        s64, smx = C.c_double(), C.c_double()
        N.call("qmt_density", handle, nx, ny, nz, h, ox, oy, oz, 1, N.PREC["fp64"], 0, C.c_void_p(q.data_ptr()),
               C.byref(s64), sh)
        N.call("qmt_density", handle, nx, ny, nz, h, ox, oy, oz, 1, prec, 0, C.c_void_p(q.data_ptr()),
               C.byref(smx), sh)
        tr = C.c_double()
        N.call("qmt_mol_trace_ps", handle, C.byref(tr), sh)
        q_raw = q.cpu().numpy()
        step()
        torch.cuda.synchronize()
        check = {"c1": {"precision": args.precision, "q_raw": q_raw, "q": q.cpu().numpy(), "v": vout.cpu().numpy(),
                        "sum_fp64": s64.value, "sum_mixed": smx.value, "two_trace_ps": 2.0 * tr.value}}
        out["batched"] = batched(basis, qmtools, N, args.precision)
        out.update(serving_streams(basis, qmtools, args.precision))
        out["c0_route"] = c0_route(basis, qmtools, N)
        out["c2_sweep"], check["c2"] = c2_sweep(basis, qmtools, N)
        out["kernels"] = other_kernels(basis, qmtools, N, hbm, ms - dens_ms, {"n3": npts, "M": 2 * nx})
    if rank == 0 and not args.no_cpu_baseline:
        out["cpu_baseline"], acc = cpu_baseline_c1(sm, basis, qmtools, check)
        if acc is not None:
            out["accuracy"] = acc
    return out


def other_kernels(basis, qmtools, N, hbm_peak, fft_ms, nfft):
    """Rooflines of the other kernels of the path (rank 0, not part of `value`)."""
    import ctypes as C
    import torch
    from qmtools import synthetic as syn
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    out = {}
    jac = {}
    for name, n, sweeps in (("c0_64^3_2000_sweeps", 64, 2000), ("c1_128^3_400_sweeps", 128, 400),
                            ("c2_192^3_200_sweeps", 192, 200)):
        npts = n ** 3
        rho = torch.rand(npts, device="cuda")
        v = torch.zeros(npts, device="cuda")
        t = torch.zeros(npts, device="cuda")
        so, d = C.c_int(), C.c_double()
        args = lambda k: (n, n, n, 0.2, C.c_void_p(rho.data_ptr()), C.c_void_p(v.data_ptr()),
                          C.c_void_p(t.data_ptr()), k, 100, 0.0, C.byref(so), C.byref(d), s)
        N.call("qmt_jacobi", *args(20))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        N.call("qmt_jacobi", *args(sweeps))
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        gbs = 12.0 * npts * sweeps / (ms / 1e3) / 1e9
        jac[name] = {"ms": ms, "us_per_sweep": 1e3 * ms / sweeps, "achieved_GBps": gbs,
                     "frac_of_hbm_peak": gbs / hbm_peak}
    out["jacobi"] = dict(jac, bytes_per_point_sweep=12,
                         kernel="qmt_jacobi (reference update), automatic kernel choice; grids up to 192^3 "
                                "(85 MB for V, T and Q) stay in the 126 MB L2, so the fraction is of the HBM "
                                "copy peak but the data is L2-resident")
    # GA single-shot automaton: 26 neighbour MLPs (4 hidden layers of 16) per voxel, 96^3 grid
    n, nl = 96, 4
    npts = n ** 3
    qube = torch.rand(2 * npts, device="cuda")
    qo = torch.empty(npts, device="cuda")
    p = ((2 * np.random.default_rng(0).random(272 * nl + 29) - 1) * 0.5).astype(np.float32)
    call = lambda: N.call("qmt_nn_singleshot", n, n, n, 0.2, C.c_void_p(qube.data_ptr()),
                          C.c_void_p(qo.data_ptr()), C.c_void_p(p.ctypes.data), int(p.size), nl, s)
    call()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(5):
        call()
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / 5
    fma = 26.0 * (272 * nl + 17)
    out["automaton_nnss_96^3_nl4"] = {"ms": ms, "voxels_per_s": npts / (ms / 1e3),
                                      "fp32_tflops": 2 * fma * npts / (ms / 1e3) / 1e12,
                                      "flop_definition": "2 x 26 x (272 NL + 17) FMA per voxel (tanh not counted)"}
    if nfft is not None:
        H = nfft["M"] ** 2 * (nfft["M"] // 2 + 1)
        fbytes = 8.0 * nfft["n3"] + 100.0 * H
        out["fft_hockney"] = {"ms": fft_ms, "algorithmic_bytes": fbytes,
                              "achieved_GBps": fbytes / (fft_ms / 1e3) / 1e9,
                              "frac_of_hbm_peak": fbytes / (fft_ms / 1e3) / 1e9 / hbm_peak,
                              "definition": "8 n^3 + 100 H bytes, H = M^2 (M/2+1), M = 2n"}
        out["gto_boundary_c1"] = gto_boundary(basis, qmtools, N, s)
        # the analytic potential on every corner of the small molecule's 64^3 grid: the
        # reference arm times its gpu_hartree_GTO on the same grid
        sm = syn.config_molecule("c0")
        mol = sm.molecule(basis, qmtools.Molecule)
        g = sm.grid(qmtools.Grid)
        nx, ny, nz, h, ox, oy, oz = g._geom()
        v = torch.zeros(nx * ny * nz, device="cuda")
        call = lambda: N.call("qmt_hartree_gto", mol.handle, nx, ny, nz, h, ox, oy, oz, C.c_void_p(v.data_ptr()), s)
        call()
        ms = _events_ms(call, 3)
        out["gto_full_grid_c0_64"] = {"ms": ms, "points": nx * ny * nz, "points_per_s": nx * ny * nz / (ms / 1e3),
                                      "precision": "FP64 McMurchie-Davidson", "points_at": "voxel corners"}
        mol.release()
    return out


def gto_boundary(basis, qmtools, N, s, reps=3):
    """The analytic potential on the medium molecule's grid boundary (the Dirichlet boundary of the
    Jacobi route): the default mixed FP32/FP64 kernels against the FP64 kernel, time and rel-L2."""
    import ctypes as C
    import torch
    from qmtools import synthetic as syn
    sm = syn.config_molecule("c1")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    nx, ny, nz, h, ox, oy, oz = g._geom()
    nb = nx * ny * nz - (nx - 2) * (ny - 2) * (nz - 2)
    res = {}
    for name, prec in (("fp64", N.PREC["fp64"]), ("mixed", N.PREC["fp32"])):
        v = torch.zeros(nx * ny * nz, device="cuda")
        N.call("qmt_set_gto_precision", prec)
        call = lambda: N.call("qmt_hartree_gto_boundary", mol.handle, nx, ny, nz, h, ox, oy, oz,
                              C.c_void_p(v.data_ptr()), s)
        call()
        res[name] = (_events_ms(call, reps), v.double().cpu().numpy())
    N.call("qmt_set_gto_precision", N.PREC["fp32"])
    # the reference's work measure: boundary points x primitive pairs of the basis functions
    # (p >= q) x ~40 flop
    almos = np.asarray(mol.ALMOs).reshape(-1, 4)
    co = np.asarray(mol.basisset.coeffs)
    npf = np.array([int(np.count_nonzero(co[int(r[3]):int(r[3]) + 20])) for r in almos], dtype=np.float64)
    pairs = 0.5 * (npf.sum() ** 2 + (npf ** 2).sum())
    flops = nb * pairs * 40.0
    ms = res["mixed"][0]
    a, b = res["mixed"][1], res["fp64"][1]
    mol.release()
    return {"ms": ms, "ms_fp64_kernel": res["fp64"][0], "boundary_points": nb, "points_per_s": nb / (ms / 1e3),
            "precision": "mixed: FP32 pair terms, FP64 for the largest pairs, near fields, atoms and sums",
            "rel_l2_vs_fp64_kernel": float(np.linalg.norm(a - b) / np.linalg.norm(b)),
            "algorithmic_flop": flops, "flop_definition": "boundary points x sum_{p>=q} nprim_p nprim_q x 40",
            "achieved_tflops": flops / (ms / 1e3) / 1e12}


TRAFFIC_JSON = ROOT / "profiles" / "density_factored_kernel_c1.traffic.json"


def profiled_traffic():
    """DRAM bytes (read + write) per launch of the factored density kernel at the bench size, from
    the machine-written summary of an ncu metrics capture (`--ncu-import`), or None."""
    if not TRAFFIC_JSON.exists():
        return None
    d = json.loads(TRAFFIC_JSON.read_text())
    return {"bytes_per_launch": d["bytes_per_launch"],
            "source": f"{TRAFFIC_JSON.name}: {d['launches']} launch(es) of {d['kernel']}, {d['command']}"}


def ncu_import(csv_path, command):
    """Writes TRAFFIC_JSON from an ncu `--csv` metrics capture of the fused density kernel
    (one row per launch and metric: ID, Kernel Name, Metric Name, Metric Unit, Metric Value)."""
    import csv
    rows = list(csv.DictReader(l for l in Path(csv_path).read_text().splitlines() if l.startswith('"')))
    scale = {"byte": 1, "Kbyte": 1e3, "Mbyte": 1e6, "Gbyte": 1e9, "KB": 1e3, "MB": 1e6, "GB": 1e9}
    per = {}
    for r in rows:
        if "density_factored_kernel" not in r["Kernel Name"]:
            continue
        if r["Metric Name"] not in ("dram__bytes_read.sum", "dram__bytes_write.sum"):
            continue
        v = float(r["Metric Value"].replace(",", "")) * scale.get(r["Metric Unit"], 1)
        per.setdefault(r["ID"], {})[r["Metric Name"]] = v
    launches = [d for d in per.values() if len(d) == 2]
    if not launches:
        raise SystemExit("no density_factored_kernel launch with both DRAM metrics in " + str(csv_path))
    rd = float(np.mean([d["dram__bytes_read.sum"] for d in launches]))
    wr = float(np.mean([d["dram__bytes_write.sum"] for d in launches]))
    out = {"kernel": "density_factored_kernel", "launches": len(launches), "dram_bytes_read": rd,
           "dram_bytes_write": wr, "bytes_per_launch": rd + wr, "command": command}
    TRAFFIC_JSON.write_text(json.dumps(out, indent=1) + "\n")
    print(json.dumps(out))


def _ref_libs():
    ref = ROOT / "oracle" / "_ref"
    paths = [ref / "utils.so", ref / "c1_bench" / "density_s1.so", ref / "c1_bench" / "fft.so"]
    return paths if all(p.exists() for p in paths) else None


def reference_hartree_kernels():
    """The reference's analytic potential (gpu_hartree_GTO) and Jacobi sweeps
    (gpu_hartree_iteration, 1000 pairs = 2000 sweeps launched back to back as its facade loop
    issues them) on the small molecule's 64^3 grid, CUDA-event timed; the bench's own arm reports
    qmt_hartree_gto and qmt_jacobi on the same grid (kernels.gto_full_grid_c0_64,
    kernels.jacobi)."""
    import ctypes as C
    import torch
    import qmtools
    from qmtools import synthetic as syn
    so_g = ROOT / "oracle" / "_ref" / "c0_64" / "hartree_gto.so"
    so_j = ROOT / "oracle" / "_ref" / "c0_64" / "hartree_iter.so"
    if not (so_g.exists() and so_j.exists()):
        return None
    lg, lj = C.CDLL(str(so_g)), C.CDLL(str(so_j))
    basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)
    sm = syn.config_molecule("c0")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    gx, gy, gz = g.GPUblocks
    n = int(g.npts)
    dev = "cuda"
    t = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a, dtype=dt).ravel()).to(dev)
    types, coords = t(mol.types, np.int32), t(mol.coords, np.float32)
    alphas, coeffs = t(basis.alphas, np.float32), t(basis.coeffs, np.float32)
    almos, dm = t(mol.ALMOs, np.int16), t(mol.dm, np.float32)
    v = torch.zeros(n, device=dev)
    vp = lambda x: C.c_void_p(x.data_ptr())
    gto = lambda: lg.ref_hartree_gto(gx, gy, gz, vp(types), vp(coords), vp(alphas), vp(coeffs), vp(almos), vp(dm),
                                     vp(v))
    assert gto() == 0
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    assert gto() == 0
    e1.record()
    torch.cuda.synchronize()
    ms_g = e0.elapsed_time(e1)
    rho = torch.rand(n, device=dev)
    a, b = torch.zeros(n, device=dev), torch.zeros(n, device=dev)
    assert lj.ref_hartree_iteration_pairs(gx, gy, gz, vp(rho), vp(a), vp(b), 10) == 0
    e0.record()
    assert lj.ref_hartree_iteration_pairs(gx, gy, gz, vp(rho), vp(a), vp(b), 1000) == 0
    e1.record()
    torch.cuda.synchronize()
    ms_j = e0.elapsed_time(e1)
    mol.release()
    return {"gto_full_grid_c0_64": {"ms": ms_g, "points": n, "points_per_s": n / (ms_g / 1e3),
                                    "kernel": "gpu_hartree_GTO (kernel_hartree.cu:288-869), FP32, voxel corners"},
            "jacobi_c0_64^3_2000_sweeps": {"ms": ms_j, "us_per_sweep": 1e3 * ms_j / 2000,
                                           "kernel": "gpu_hartree_iteration (kernel_hartree.cu:85-171), "
                                                     "2 launches per pair, no host synchronisation"}}


def run_reference_gpu(args, world, rank, local, paths):
    """The reference path on the same B200: its density kernel (kernel_density.cu), grid total
    and rescale (kernel_utils.cu) and the periodic FFT route (kernel_fft.cu around cuFFT), with
    the launch shapes and host steps of its facade (Compute_density, Compute_hartree_fft)."""
    import ctypes as C
    import torch
    import qmtools
    from qmtools import synthetic as syn
    qmtools.set_verbose(False)
    torch.cuda.set_device(local)
    ut, dl, fl_ = (C.CDLL(str(p)) for p in paths)
    basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)
    sm = syn.config_molecule("c1")
    mol = sm.molecule(basis, qmtools.Molecule)
    g = sm.grid(qmtools.Grid)
    nx, ny, nz = g.space_shape()
    gx, gy, gz = g.GPUblocks
    n = nx * ny * nz
    h = float(g.step)
    ox, oy, oz = (float(g.origin[k]) for k in "xyz")
    dev = "cuda"
    pin = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a, dtype=dt).ravel()).pin_memory()
    coords_h, dm_h = pin(mol.coords, np.float32), pin(mol.dm, np.float32)
    coords, dm = coords_h.to(dev), dm_h.to(dev)
    types = torch.from_numpy(np.ascontiguousarray(mol.types, dtype=np.int32)).to(dev)
    almos = torch.from_numpy(np.ascontiguousarray(mol.ALMOs, dtype=np.int16)).to(dev)
    alphas = torch.from_numpy(np.ascontiguousarray(basis.alphas, dtype=np.float32)).to(dev)
    coeffs = torch.from_numpy(np.ascontiguousarray(basis.coeffs, dtype=np.float32)).to(dev)
    q = torch.zeros(n, device=dev)
    tot = torch.zeros(1, device=dev)
    wr, c1, c2, v = (torch.zeros(k * n, device=dev) for k in (1, 2, 2, 1))
    v_h = torch.empty(n, dtype=torch.float32).pin_memory()
    vp = lambda t: C.c_void_p(t.data_ptr())
    f = C.c_float

    def step(e2e=False):
        if e2e:
            coords.copy_(coords_h, non_blocking=True)
            dm.copy_(dm_h, non_blocking=True)
        assert dl.ref_density(gx, gy, gz, f(h), f(ox), f(oy), f(oz), vp(coords), vp(alphas), vp(coeffs), vp(almos),
                              vp(dm), vp(q)) == 0
        assert ut.ref_total(gx, gy, gz, vp(q), vp(tot)) == 0
        factor = np.float32(mol.qtot / float(tot.item()))
        assert ut.ref_rescale(gx, gy, gz, vp(q), f(factor)) == 0
        assert fl_.ref_fft_route(gx, gy, gz, nx, ny, nz, vp(q), vp(types), vp(coords), vp(wr), vp(c1), vp(c2),
                                 vp(v)) == 0
        if e2e:
            v_h.copy_(v)
        torch.cuda.synchronize()

    def timed(k, e2e, budget_s):
        # up to k steps, stopping once budget_s of wall time is spent (a reference step takes
        # seconds): the run stays within a few minutes at any --steps
        ts = []
        t_start = time.perf_counter()
        for _ in range(k):
            t0 = time.perf_counter()
            step(e2e)
            ts.append(time.perf_counter() - t0)
            if time.perf_counter() - t_start > budget_s:
                break
        return float(np.mean(ts)), len(ts)

    nwarm = min(args.warmup, 3)   # a reference step takes seconds
    for _ in range(nwarm):
        step()
    ms, nsteps = timed(args.steps, False, 60.0)
    e2e_ms, _ = timed(max(1, args.steps // 2), True, 30.0)
    ms *= 1000.0
    e2e_ms *= 1000.0
    v_ = n / (ms / 1000.0)
    hk = reference_hartree_kernels()
    return {"metric": METRIC, "value": v_, "unit": UNIT, "n_gpus": world, "steps": nsteps, "warmup": nwarm,
            "ms_per_step": ms, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "fp32",
            "data": "synthetic", "impl": "reference",
            "config": {"workload": WORKLOAD.replace("density + Hockney FFT Poisson on 256^3",
                                                   "density + periodic FFT Poisson on 128^3 (the reference's solve)"),
                       "grid_pts_per_step": n, "timing": "host wall clock around each synchronised step; up to --steps steps within 60 s (end to end: 30 s)"},
            "cpu_baseline": {"value": v_, "unit": UNIT, "cores": 0, "kind": "reference",
                             "sample": "the full step on the GPU: the reference's kernels compiled from its sources "
                                       "for sm_100a (oracle/_ref/c1_bench), no host cores used"},
            "e2e": {"value": n / (e2e_ms / 1000.0), "unit": UNIT,
                    "h2d_bytes_per_step": int(4 * (coords_h.numel() + dm_h.numel())), "d2h_bytes_per_step": 4 * n},
            "hartree_kernels": hk}


def run_reference(args, world, rank, local, pg):
    """The reference's implementation of this path, timed on the same workload (rank 0 only)."""
    if rank != 0:
        return None
    paths = _ref_libs()
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except Exception:
        has_gpu = False
    if paths is not None and has_gpu:
        return run_reference_gpu(args, world, rank, local, paths)
    import qmtools
    from qmtools import synthetic as syn
    qmtools.set_verbose(False)
    basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)
    sm = syn.config_molecule("c1")
    # CPU oracle port of the reference algorithm (FP64 density + FFT solve)
    samples = []
    for _ in range(args.warmup):
        cpu_baseline_c1(sm, basis, qmtools)
    for _ in range(args.steps):
        samples.append(cpu_baseline_c1(sm, basis, qmtools)[0])
    v = float(np.median([s["value"] for s in samples]))
    cb = dict(samples[0])
    cb["value"] = v
    return {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1000.0 * (128 ** 3) / v, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "fp64", "data": "synthetic", "impl": "reference",
            "config": {"workload": WORKLOAD},
            "cpu_baseline": cb, "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "note": "FP64 CPU port of the reference algorithm on the host cores (reference kernel builds absent)"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="fp16x3")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--quick", action="store_true", help="headline step only (no plain-FP32, batch, serving)")
    ap.add_argument("--grid", type=int, default=0, help="cube edge of a smaller grid for the same molecule")
    ap.add_argument("--only", default="", choices=["", "jacobi", "gto"], help="run one kernel family alone (profiling)")
    ap.add_argument("--ncu-import", default="", help="ncu --csv metrics capture of the factored density kernel "
                                                     "to summarise into profiles/ (no GPU needed)")
    ap.add_argument("--ncu-command", default="", help="the command line of that capture (recorded beside it)")
    args = ap.parse_args()
    if args.ncu_import:
        ncu_import(args.ncu_import, args.ncu_command)
        return
    args.warmup = max(args.warmup, 3)
    world, rank, local, pg = dist_setup()
    if args.only == "jacobi":
        # the Jacobi solve alone (64^3 for 2000 sweeps, 128^3 for 400): its profiling case
        import torch
        import qmtools
        from qmtools import _native as N
        qmtools.set_verbose(False)
        torch.cuda.set_device(local)
        N.ensure_device(None)
        print(json.dumps(other_kernels(None, qmtools, N, peaks()[1], 0.0, None)["jacobi"]))
        return
    if args.only == "gto":
        # the analytic boundary potential alone (FP64 kernel once, then the mixed kernels
        # 1 + reps times): its profiling case
        import ctypes as C
        import torch
        import qmtools
        from qmtools import _native as N
        qmtools.set_verbose(False)
        torch.cuda.set_device(local)
        N.ensure_device(None)
        basis = qmtools.BasisSet(qmtools.BASIS_CCPVDZ)
        print(json.dumps(gto_boundary(basis, qmtools, N, C.c_void_p(torch.cuda.current_stream().cuda_stream))))
        return
    try:
        if args.impl == "reference":
            out = run_reference(args, world, rank, local, pg)
        else:
            out = run_ours(args, world, rank, local, pg)
        if rank == 0 and out is not None:
            print(json.dumps(out))
    finally:
        if pg is not None:
            pg.destroy_process_group()


if __name__ == "__main__":
    main()
