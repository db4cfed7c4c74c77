"""Benchmark: pressure projections per second to FP64 relative residual 1e-6 on
the 384x384x256 pot (dx = 0.5 mm).

One step = one full projection of the reference's pressure_projection
(python/boilingsim/fluid.py:612-734) with the to-tolerance solver: restore
the pre-projection velocities, divergence, solve A p = b to
||b - A p||_2 <= 1e-6 ||b||_2 (FP64 residual of the FP64 iterate), gradient
subtract, diagnostic max|div| on the device.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--storage fp32|fp16|bf16]

N > 1 runs N independent replicas (one per GPU, launched by torchrun); the
path does not shard, so there is no collective on the data path.  Prints one
JSON line on rank 0.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "boiling-sim_b200"))

METRIC = "projections/s to rel-residual 1e-6 at 384²×256: learned+mixed vs plain FP32"
DX, DT, RHO, TOL, SEED = 0.0005, 0.01, 997.0, 1e-6, 7
WORKLOAD = ("pot 384x384x256 dx=0.5mm (R_in 168, wall 12, water line 213, carrot r36 L180), "
            "velocities N(0,0.05) box-smoothed 3x + plume 0.1 m/s seed 7, full projection to "
            "FP64 rel-residual 1e-6")
# Iterations the reference's Jacobi-preconditioned CG needs to meet its own
# stopping rule (recursive ||r|| < 1e-6 ||b||, checked every 5 iterations from
# iteration 8) on this workload; measured with this library's reference-
# compatible pressure_solve_pcg_launch (same algorithm) when a GPU is present.
REF_PCG_ITERS_FALLBACK = 1281
# DRAM traffic per launch measured by ncu (dram__bytes_read.sum + dram__bytes_write.sum) of the
# dominant kernel class at 384x384x256: the fused CG update + restriction with FP16 storage
# (286.2 + 119.6 MB; algorithmic 427.3 MB).
CAPTURED_TRAFFIC = {("cg_update_restrict_fine", "fp16"): 405_800_000}


def max_over_ranks(ms: float, dist, device) -> float:
    """The slowest replica's time; every rank takes part (the same collective
    on every rank, in the same order).  Without a process group: ms itself."""
    if dist is None:
        return ms
    import torch

    t = torch.tensor([float(ms)], device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def job_rate(world: int, units_per_rank: float, ms: float) -> float:
    """Whole-job units per second: `world` replicas each process
    units_per_rank in ms (the max over ranks)."""
    return world * units_per_rank * 1e3 / ms


def _peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def active_tile_cells(mat, nsm: int) -> int:
    """Cells in the level-0 column tiles that hold a fluid cell: tiles of 8 j
    rows x 128 k x bi i planes, bi the largest even value <= 16 that still
    gives two tiles per SM (the library's tiling rule)."""
    nx, ny, nz = mat.shape
    cols = ((nz // 4 + 31) // 32) * ((ny + 7) // 8)
    bi = 16
    while bi > 2 and cols * ((nx + bi - 1) // bi) < 2 * nsm:
        bi -= 2
    f = mat == 0
    total = 0
    for i0 in range(0, nx, bi):
        fi = f[i0:i0 + bi]
        for j0 in range(0, ny, 8):
            fj = fi[:, j0:j0 + 8]
            for k0 in range(0, nz, 128):
                blk = fj[:, :, k0:k0 + 128]
                if blk.any():
                    total += blk.size
    return int(total)


def _workload():
    from boilingsim_b200 import scenes as S

    mat = S.pot_mat(S.POT_384)
    ux, uy, uz = S.velocity_field(mat, seed=SEED)
    return mat, ux, uy, uz


class Clocks:
    """SM clock and clock-event reasons sampled every 10 ms during the timed
    region (NVML reads from a background thread; nvidia-smi at 100 ms when
    NVML is not importable).  Reads only: no clock or power setting changes."""

    # NVML clock-event reason bits
    REASONS = {0x8: "hw_slowdown", 0x40: "hw_thermal_slowdown", 0x20: "sw_thermal_slowdown",
               0x4: "sw_power_cap"}

    def __init__(self, index: int):
        import threading

        self.samples, self.max_mhz, self.reasons = [], 0.0, set()
        self.proc = None
        self.stop_ev = threading.Event()
        try:
            import pynvml

            pynvml.nvmlInit()
            self.nvml = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM))
            self.thread = threading.Thread(target=self._run, daemon=True)
            self.thread.start()
            return
        except Exception:
            self.nvml = None
        self.path = f"/tmp/bsp_clocks_{os.getpid()}.csv"
        q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def _run(self):
        nv = self.nvml
        while not self.stop_ev.is_set():
            try:
                self.samples.append(float(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM)))
                bits = nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)
                for b, nm in self.REASONS.items():
                    if bits & b:
                        self.reasons.add(nm)
            except Exception:
                pass
            self.stop_ev.wait(0.01)

    def stop(self):
        if self.nvml is not None:
            self.stop_ev.set()
            self.thread.join(timeout=2)
            sm = self.samples
            if not sm:
                return None
            load = [x for x in sm if x > 0.5 * max(sm)] or sm
            return {"sm_mhz": float(np.median(load)), "sm_max_mhz": self.max_mhz,
                    "reasons": sorted(self.reasons), "samples": len(sm), "source": "nvml, 10 ms"}
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = max(mx, float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return None
        load = [s for s in sm if s > 0.5 * max(sm)] or sm
        return {"sm_mhz": float(np.median(load)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm), "source": "nvidia-smi, 100 ms"}


def cpu_reference(mat, ux, uy, uz, ref_iters):
    """The reference's projection algorithm (divergence, Jacobi-PCG to its own
    stopping rule, gradient subtract, diagnostic divergence) restated in C
    (oracle/, OpenMP on all host threads), timed on a bounded sample: the
    divergence/gradient passes once and PCG iterations 2 -> 12 on the full
    workload; projections/s = 1 / (t_div + ref_iters * t_iter + t_grad + t_div)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O

    threads = os.cpu_count() or 1
    O.set_threads(threads)
    t0 = time.perf_counter()
    div = O.divergence(ux, uy, uz, mat, DX)
    t_div = time.perf_counter() - t0
    t0 = time.perf_counter()
    O.pcg(div, mat, DX, DT, RHO, 1e-30, 2)
    t2 = time.perf_counter() - t0
    t0 = time.perf_counter()
    O.pcg(div, mat, DX, DT, RHO, 1e-30, 12)
    t12 = time.perf_counter() - t0
    t_iter = max(t12 - t2, 1e-9) / 10.0
    p = np.zeros(mat.shape, np.float32)
    t0 = time.perf_counter()
    O.subtract_gradient(ux, uy, uz, p, mat, DX, DT, RHO)
    t_grad = time.perf_counter() - t0
    t_proj = 2 * t_div + ref_iters * t_iter + t_grad
    return {"value": 1.0 / t_proj, "unit": "projections/s", "cores": threads, "kind": "port",
            "sample": (f"full 384x384x256 workload: divergence and gradient once, PCG iterations "
                       f"2->12 timed ({t_iter*1e3:.1f} ms/iteration); projection = "
                       f"{ref_iters} PCG iterations (the reference's stopping rule at tol 1e-6)"),
            "s_per_projection": t_proj}


def cell_classes_t(mat_t):
    """int8 device tensor: 0 fluid, 1 air, 2 solid (every other material id)."""
    import torch

    return torch.where(mat_t == 0, 0, torch.where(mat_t == 2, 1, 2)).to(torch.int8)


def apply_A_f64(p64, cls):
    """(A p)_c = 6 p_c - sum g(n) on fluid cells in FP64 on the device (the
    operator of laplacian_spmv.cu:62-143: neighbour fluid -> p_n, air or
    outside the grid -> 0, solid -> p_c); 0 elsewhere.  Measurement plumbing
    for residuals of iterates that live in FP32."""
    import torch

    fl = cls == 0
    s = torch.zeros_like(p64)
    for dim in range(3):
        for sh in (1, -1):
            pn = torch.roll(p64, sh, dim)
            cn = torch.roll(cls, sh, dim)
            edge = [slice(None)] * 3
            edge[dim] = 0 if sh == 1 else -1
            cn[tuple(edge)] = 1  # beyond the grid: air
            s += torch.where(cn == 0, pn, torch.where(cn == 2, p64, torch.zeros_like(p64)))
    return torch.where(fl, 6.0 * p64 - s, torch.zeros_like(p64))


def plain_fp32_to_tolerance(mat_t, mask, div, solver, dev, sweeps=8000, chunk=2000):
    """The plain FP32 Jacobi drop-in (fluid.py:689-701, jacobi_pressure.cu:
    228-270) run to the projection's tolerance, ||b - A p|| <= 1e-6 ||b||
    (config.py:166-176) -- extrapolated, because at 384x384x256 it needs on
    the order of 10^5-10^6 sweeps.

    Measured: `sweeps` sweeps from p = 0 (event-timed per sweep), with the
    FP64 relative residual every `chunk` sweeps.  A Jacobi sweep is p <- p +
    (b - A p)/6 (the update (s - rhs)/6 rewritten), so its error contracts in
    the end by rho = 1 - lambda_min/6 per sweep, lambda_min the smallest
    eigenvalue of A on the fluid cells; lambda_min is measured by inverse
    iteration with the library's tolerance solver (8 steps, Rayleigh
    quotient).  Sweeps to tolerance = sweeps + ln(1e-6 / r_sweeps) / ln(rho).
    Also reported: the FP32 rounding floor, the relative residual of the
    converged FP64 pressure rounded to float -- the plain FP32 iteration
    cannot go below it."""
    import math

    import torch

    from boilingsim_b200 import _lib

    nx, ny, nz = mat_t.shape
    cls = cell_classes_t(mat_t)
    fl = cls == 0
    b = -(float(np.float32(RHO)) * float(np.float32(DX)) ** 2 / float(np.float32(DT))) * \
        torch.where(fl, div.double(), torch.zeros((), dtype=torch.float64, device=dev))
    bn = float(torch.linalg.norm(b))

    def rel(p32):
        return float(torch.linalg.norm(b - apply_A_f64(p32.double(), cls))) / bn

    p = torch.zeros_like(div)
    q = torch.empty_like(div)
    rhs = torch.empty_like(div)
    hist = []
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    ms = 0.0
    done = 0
    while done < sweeps:
        n = min(chunk, sweeps - done)
        torch.cuda.synchronize()
        ev[0].record()
        # a fresh call each chunk continues from p (the first call starts from 0)
        _lib.call("bsp_jacobi_solve", _lib.ptr(p), _lib.ptr(q), _lib.ptr(div), _lib.ptr(rhs),
                  _lib.ptr(mask), nx, ny, nz, DX, DT, RHO, n, 1, _lib.stream_handle())
        ev[1].record()
        torch.cuda.synchronize()
        ms += ev[0].elapsed_time(ev[1])
        done += n
        hist.append([done, rel(p)])
    ms_sweep = ms / sweeps
    # smallest eigenvalue of A on the fluid cells: inverse iteration
    g = torch.Generator(device=dev).manual_seed(SEED)
    v = torch.where(fl, torch.rand(mat_t.shape, generator=g, device=dev, dtype=torch.float64),
                    torch.zeros((), dtype=torch.float64, device=dev))
    lam = float("nan")
    to_div = -float(np.float32(DT)) / (float(np.float32(RHO)) * float(np.float32(DX)) ** 2)
    x = torch.zeros_like(div)
    for _ in range(8):
        v = v / torch.linalg.norm(v)
        d = (v * to_div).float().contiguous()  # so that b = v
        solver.solve(d, DX, DT, RHO, tol=1e-9, p=x, raise_on_fail=False)
        w = solver.last.p64_dev.clone()
        lam = float((v * v).sum() / (v * w).sum())  # (v.v) / (v.A^-1 v)
        v = torch.where(fl, w, torch.zeros_like(w))
    rho_j = 1.0 - lam / 6.0
    r_t = hist[-1][1]
    remaining = math.log(TOL / r_t) / math.log(rho_j) if r_t > TOL else 0.0
    total = sweeps + remaining
    obs = (hist[-1][1] / hist[-2][1]) ** (1.0 / chunk) if len(hist) >= 2 else float("nan")
    # FP32 floor: the converged FP64 pressure rounded to float
    solver.solve(div, DX, DT, RHO, tol=1e-10, p=x, raise_on_fail=False)
    floor = rel(solver.last.p64_dev.float())
    return {"sweeps_measured": sweeps, "ms_per_sweep": round(ms_sweep, 5),
            "rel_residual_history": [[n, float(f"{r:.4e}")] for n, r in hist],
            "lambda_min": lam, "asymptotic_rate_per_sweep": rho_j,
            "observed_rate_last_chunk": obs,
            "sweeps_to_tol_extrapolated": round(total),
            "fp32_rounding_floor_rel_residual": floor,
            "reaches_tol_in_fp32": bool(floor <= TOL),
            "method": "extrapolated: measured sweeps + ln(1e-6/r)/ln(1 - lambda_min/6)"}


def reference_cuda_block(mat_t, div, dev, ours_sweep_ms, ours_pcg):
    """The reference's own CUDA (crates/cuda-kernels/src, compiled from source
    into oracle/_ref/libref_fma.so with its default flags) timed on this GPU
    beside this library, on the same 384x384x256 workload: the fused Jacobi
    solve of 200 sweeps (pressure_solve_launch, jacobi_pressure.cu:228-270)
    and the Jacobi-PCG to its tolerance 1e-6 (pressure_solve_pcg_launch,
    pressure_solve_pcg.cu:89-243).  A baseline leg, like cpu_baseline."""
    import ctypes

    import torch

    path = os.path.join(ROOT, "oracle", "_ref", "libref_fma.so")
    if not os.path.exists(path):
        return {"unavailable": "oracle/_ref/libref_fma.so not built (reference sources absent "
                               "when the library was built)"}
    L = ctypes.CDLL(path)
    P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
    L.pressure_solve_launch.argtypes = [P, P, P, P, I, I, I, F, F, F, I, I, I]
    L.pressure_solve_launch.restype = I
    L.pressure_solve_pcg_launch.argtypes = [P, P, P, I, I, I, F, F, F, I, I, F, I] + [P] * 13 + \
        [ctypes.POINTER(I)]
    L.pressure_solve_pcg_launch.restype = I
    nx, ny, nz = mat_t.shape
    p = torch.zeros_like(div)
    q = torch.zeros_like(div)
    out = {"library": "oracle/_ref/libref_fma.so (reference sources, default nvcc flags, "
                      "sm_100a)"}
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    # legacy default stream: record the events on it
    s0 = torch.cuda.default_stream(dev)
    assert L.pressure_solve_launch(p.data_ptr(), q.data_ptr(), div.data_ptr(), mat_t.data_ptr(),
                                   nx, ny, nz, DX, DT, RHO, 20, 0, 2) == 0
    torch.cuda.synchronize()
    ev[0].record(s0)
    rc = L.pressure_solve_launch(p.data_ptr(), q.data_ptr(), div.data_ptr(), mat_t.data_ptr(),
                                 nx, ny, nz, DX, DT, RHO, 200, 0, 2)
    ev[1].record(s0)
    torch.cuda.synchronize()
    ref_ms = ev[0].elapsed_time(ev[1])
    out["jacobi_200_sweeps"] = {"reference_ms": round(ref_ms, 3), "status": rc,
                                "ours_ms": round(200 * ours_sweep_ms, 3),
                                "speedup": round(ref_ms / (200 * ours_sweep_ms), 2)}
    ws = [torch.zeros(mat_t.shape, device=dev) for _ in range(5)] + \
        [torch.zeros(1024, device=dev)] + [torch.zeros(1, device=dev) for _ in range(7)]
    it = ctypes.c_int(0)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    rc = L.pressure_solve_pcg_launch(p.data_ptr(), div.data_ptr(), mat_t.data_ptr(), nx, ny, nz,
                                     DX, DT, RHO, 0, 2, TOL, 5000, *[w.data_ptr() for w in ws],
                                     ctypes.byref(it))
    torch.cuda.synchronize()
    ref_pcg_ms = (time.perf_counter() - t0) * 1e3  # host-synchronising launcher: host clock
    cls = cell_classes_t(mat_t)
    fl = cls == 0
    b = -(float(np.float32(RHO)) * float(np.float32(DX)) ** 2 / float(np.float32(DT))) * \
        torch.where(fl, div.double(), torch.zeros((), dtype=torch.float64, device=dev))
    true_rel = float(torch.linalg.norm(b - apply_A_f64(p.double(), cls)) / torch.linalg.norm(b))
    out["pcg_to_1e-6"] = {"reference_ms": round(ref_pcg_ms, 2), "iterations": it.value,
                          "status": rc, "true_rel_residual_fp64": true_rel,
                          "note": "the reference stops on its recursive FP32 residual; the "
                                  "true residual of its answer is given beside"}
    out["pcg_to_1e-6"].update(ours_pcg)
    return out


COND_SWEEPS = 50  # diffusion_max_iter of the reference's scenario files


def conduction_bench(mat, dev, peak, peak_kind, cpu: bool):
    """Backward-Euler conduction on the same 384x384x256 pot (steel pot, water,
    carrot, air; thermal.py:259-388, 647-658): one conduction step = the
    snapshot + COND_SWEEPS Jacobi sweeps, event-timed; the sweep kernels alone
    (on cell classes, and on uint8 material ids) event-timed over 40 ping-pong
    launches each.  Algorithmic
    bytes per sweep = 1 B of material id per cell + 12 B (T_iter, T_old, store)
    per non-air cell -- air cells are neither read nor written, as in the
    reference kernel.  Fields total 490 MB (> 126 MB L2)."""
    import torch

    from boilingsim_b200 import _lib
    from boilingsim_b200 import thermal as TH

    nx, ny, nz = mat.shape
    n = mat.size
    n_solid = int((mat != TH.MAT_AIR).sum())
    rng = np.random.default_rng(SEED)
    base = np.array([330.0, 380.0, 295.15, 300.0], np.float32)[mat]
    T0 = (base + rng.standard_normal(mat.shape).astype(np.float32)).astype(np.float32)
    props = TH.MaterialProps.from_materials("steel_304", device=dev)
    grid = TH.ThermalGrid(nx, ny, nz, DX, torch.as_tensor(T0).to(dev),
                          torch.as_tensor(mat).to(dev))
    grid.mat_id = TH.material_ids(grid.mat)
    grid.classes = TH.cell_classes(grid.mat) or False
    ws = TH.allocate_thermal_workspace(grid, device=dev)
    cfg = TH.ThermalConfig()
    cfg.solver.diffusion_max_iter = COND_SWEEPS
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(3):
        TH.implicit_conduction_step(grid, props, ws, cfg, DT)
    reps = 5
    torch.cuda.synchronize()
    e0.record(stream)
    for _ in range(reps):
        TH.implicit_conduction_step(grid, props, ws, cfg, DT)
    e1.record(stream)
    torch.cuda.synchronize()
    step_ms = e0.elapsed_time(e1) / reps
    a, b = grid.T, ws.T_iter_alt
    common = [nx, ny, nz, _lib.ptr(props.k_wp), _lib.ptr(props.rho_wp), _lib.ptr(props.cp_wp), 4,
              DX, DT, 10.0, 295.15]

    def time_sweeps(fn, lead, tail, sweeps=40):
        for it in range(4 + sweeps):
            if it == 4:
                torch.cuda.synchronize()
                e0.record(stream)
            _lib.call(fn, _lib.ptr(b if it % 2 == 0 else a), _lib.ptr(a if it % 2 == 0 else b),
                      _lib.ptr(ws.T_old_snapshot), *lead, *common, *tail, _lib.stream_handle())
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / sweeps

    def sweep_entry(kernel, ms_):
        g = alg / (ms_ * 1e-3) / 1e9
        return {"kernel": kernel, "ms": round(ms_, 5), "algorithmic_bytes": int(alg),
                "non_air_cells": n_solid, "GB/s": round(g, 1), "peak": peak,
                "peak_source": peak_kind, "frac": round(g / peak, 4)}

    alg = n + 12.0 * n_solid
    ms_ids = time_sweeps("bsp_conduction_sweep_u8", [_lib.ptr(grid.mat_id)], [TH.MAT_AIR])
    out = {"workload": "pot 384x384x256 dx=0.5mm, steel pot / water / carrot / air, dt 0.01 s, "
                       f"{COND_SWEEPS} backward-Euler Jacobi sweeps per step",
           "steps_per_s": round(1e3 / step_ms, 2), "ms_per_step": round(step_ms, 4),
           "gpu_launches_per_step": COND_SWEEPS + (COND_SWEEPS % 2)}
    c = grid.classes
    if c:
        ms_cls = time_sweeps("bsp_conduction_sweep_cls",
                             [_lib.ptr(c.cls), _lib.ptr(c.patterns), c.n_classes,
                              _lib.ptr(c.tiles)],
                             [TH.MAT_AIR])
        out["sweep"] = sweep_entry("be_cls_tma_kernel" if nz % 16 == 0 else "be_cls_col_kernel",
                                   ms_cls)
        out["cell_classes"] = c.n_classes
        out["sweep_material_ids"] = sweep_entry("be_col_kernel", ms_ids)
    else:
        out["sweep"] = sweep_entry("be_col_kernel", ms_ids)
    if cpu:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O

        threads = os.cpu_count() or 1
        O.set_threads(threads)
        hp = (props.k, props.rho, props.c_p)
        t0 = time.perf_counter()
        O.conduction_sweep(T0, T0, T0, mat, hp, DX, DT, 10.0, 295.15)
        t_sweep = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": round(1.0 / (COND_SWEEPS * t_sweep), 4),
                               "unit": "conduction steps/s", "cores": threads, "kind": "port",
                               "sample": f"one full-grid sweep of the C restatement "
                                         f"({t_sweep*1e3:.0f} ms) x {COND_SWEEPS}"}
    return out


def advection_bench(mat, ux, uy, uz, dev, peak, peak_kind, cpu: bool):
    """Semi-Lagrangian advect_all (fluid.py:737-776) on the 384x384x256 pot with
    the workload's velocities, dt 0.01 s, origin (-nx dx/2, -ny dx/2, -4 dx):
    event-timed over 5 calls after 2 untimed, with the reference's copy back
    into the grid and without it (results left in the workspace).
    Algorithmic bytes per call without the copy: read ux, uy, uz, T, mask,
    T_ext (4+4+4+4+1+4 per cell); write the three velocity buffers, T_ext and
    T_tmp (12+4+4) = 41 B/cell; the copy back adds 32 B/cell."""
    import torch

    from boilingsim_b200 import _lib
    from boilingsim_b200 import fluid as F

    nx, ny, nz = mat.shape
    n = mat.size
    rng = np.random.default_rng(SEED)
    T0 = (330.0 + rng.standard_normal(mat.shape)).astype(np.float32)
    org = (-nx * DX / 2, -ny * DX / 2, -4 * DX)
    mask = F.cell_mask(torch.as_tensor(mat).to(dev))
    fields = [torch.as_tensor(a).to(dev) for a in (ux, uy, uz, T0)]
    tmp = [torch.empty_like(a) for a in fields]
    ext = torch.empty_like(fields[3])
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def run(copy_back):
        _lib.call("bsp_advect_all", *(_lib.ptr(a) for a in (*fields, *tmp, ext, mask)), nx, ny,
                  nz, *org, DX, DT, copy_back, _lib.stream_handle())

    out = {"workload": "pot 384x384x256 dx=0.5mm, workload velocities (plume 0.1 m/s), "
                       "T 330 K + N(0,1), dt 0.01 s, advect_all"}
    for cb, key in ((0, "no_copy"), (1, "with_copy_back")):
        for _ in range(2):
            run(cb)
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(5):
            run(cb)
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / 5
        alg = (41.0 + 32.0 * cb) * n
        g = alg / (ms * 1e-3) / 1e9
        out[key] = {"ms": round(ms, 4), "algorithmic_bytes": int(alg), "GB/s": round(g, 1),
                    "peak": peak, "peak_source": peak_kind, "frac": round(g / peak, 4)}
    out["calls_per_s"] = round(1e3 / out["with_copy_back"]["ms"], 2)
    out["gpu_launches_per_call"] = 2  # the extension and the march
    if cpu:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O

        threads = os.cpu_count() or 1
        O.set_threads(threads)
        t0 = time.perf_counter()
        O.advect_all(ux, uy, uz, T0, mat, org, DX, DT)
        t = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": round(1.0 / t, 4), "unit": "advect_all calls/s",
                               "cores": threads, "kind": "port",
                               "sample": f"one full-grid advect_all of the C restatement "
                                         f"({t*1e3:.0f} ms)"}
    return out


def run_learned(args, dev, rank, world, dist):
    """Learned warm start at 192x192x128 (walls 2/3/4 cells, plume 0.02 / 0.1 /
    0.3 m/s): the trained U-Net's pressure starts the solve, which finishes to
    FP64 rel-residual 1e-6.  Per scene: inner iterations cold and warm, the
    network's relative error against the converged pressure, the prediction
    and solve times (CUDA events).  value = projections/s of prediction +
    warm solve; the plain line is the cold solve of the same storage."""
    import torch

    from boilingsim_b200 import learned as LR
    from boilingsim_b200 import scenes as S

    net = LR.UNet.load(device=dev)
    rows = []
    for tw in (2, 3, 4):
        for plume in (0.02, 0.1, 0.3):
            for r in LR.evaluate(net, S.pot_192(tw), seeds=(SEED,), plume=plume,
                                 storage=args.storage):
                r.update({"wall": tw, "plume": plume})
                rows.append(r)
    ms_learned = float(np.mean([r["predict_ms"] + r["warm_ms"] for r in rows]))
    ms_plain = float(np.mean([r["cold_ms"] for r in rows]))
    if rank == 0:
        line = {
            "metric": "projections/s (solve) to rel-residual 1e-6 at 192x192x128, learned warm "
                      "start vs the same solve from zero",
            "value": round(1e3 / ms_learned, 3), "unit": "projections/s", "n_gpus": world,
            "higher_is_better": True, "dtype": "bf16 network / f32 solve",
            "data": "synthetic", "config": {"workload": "pot_192 walls 2/3/4, plumes "
                                                        "0.02/0.1/0.3 m/s, seed 7",
                                            "storage": args.storage},
            "plain_projections_per_s": round(1e3 / ms_plain, 3),
            "inner_iterations_cold_mean": float(np.mean([r["cold_inner"] for r in rows])),
            "inner_iterations_warm_mean": float(np.mean([r["warm_inner"] for r in rows])),
            "net_rel_error_mean": float(np.mean([r["net_rel_error"] for r in rows])),
            "predict_ms_mean": float(np.mean([r["predict_ms"] for r in rows])),
            "rows": rows,
        }
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


def run_batched(args, dev, rank, world, dist):
    """64 pot instances of uneven sizes (seeded draw, 48^3 .. 128x128x96), each
    with its own seeded velocity field, solved FP32-stored to FP64 rel-residual
    1e-6 in cooperative launches of up to 24; compared with 64 sequential host-driven
    solves of the same instances.  value = instances/s of the batched launch."""
    import torch

    from boilingsim_b200 import fluid as F
    from boilingsim_b200 import scenes as S
    from boilingsim_b200.solver import BatchSolver, TolSolver

    specs = S.random_batch_specs(64, seed=SEED)
    masks, divs, ps = [], [], []
    cells = 0
    for spec, seed in specs:
        mat = S.pot_mat(spec)
        ux, uy, uz = S.velocity_field(mat, seed=seed)
        m = F.cell_mask(torch.as_tensor(mat).to(dev))
        d = torch.zeros(mat.shape, dtype=torch.float32, device=dev)
        F.compute_divergence(d, *[torch.as_tensor(a).to(dev) for a in (ux, uy, uz)], m, 0.002)
        masks.append(m)
        divs.append(d)
        ps.append(torch.zeros_like(d))
        cells += mat.size
    batch = BatchSolver(masks, args.storage)
    infos = batch.solve(divs, ps, 0.002, DT, RHO, tol=TOL)  # builds the setups
    for _ in range(max(0, args.warmup - 1)):
        batch.solve(divs, ps, 0.002, DT, RHO, tol=TOL, wait=False)
    torch.cuda.synchronize()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record()
    for _ in range(args.steps):
        batch.solve(divs, ps, 0.002, DT, RHO, tol=TOL, wait=False)
    ev1.record()
    torch.cuda.synchronize()
    ms = ev0.elapsed_time(ev1) / args.steps
    infos = batch.solve(divs, ps, 0.002, DT, RHO, tol=TOL)
    worst = max(i.rel_residual for i in infos)
    # sequential host-driven solves of the same 64 instances
    singles = [TolSolver(m, args.storage) for m in masks]
    for s_, d, p in zip(singles, divs, ps):
        s_.solve(d, 0.002, DT, RHO, tol=TOL, p=p)
    torch.cuda.synchronize()
    ev0.record()
    for _ in range(max(1, args.steps // 2)):
        for s_, d, p in zip(singles, divs, ps):
            s_.solve(d, 0.002, DT, RHO, tol=TOL, p=p)
    ev1.record()
    torch.cuda.synchronize()
    seq_ms = ev0.elapsed_time(ev1) / max(1, args.steps // 2)
    ms = max_over_ranks(ms, dist, dev)
    if rank == 0:
        print(json.dumps({
            "metric": "instances/s, 64 uneven pot scenes to FP64 rel-residual 1e-6",
            "value": round(job_rate(world, 64, ms), 2), "unit": "instances/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms, 3),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic",
            "config": {"workload": f"64 pot scenes, sizes 48^3..128x128x96 (seed {SEED}), "
                                   f"{cells} cells in total, dx 2 mm", "storage": args.storage,
                       "launch": "one cooperative launch per 24 instances (a group of CTAs each)"},
            "sequential_host_driven": {"value": round(64e3 / seq_ms, 2), "unit": "instances/s",
                                       "ms_per_64": round(seq_ms, 3)},
            "worst_rel_residual_fp64": worst,
            "inner_iterations": [i.inner_iterations for i in infos][:8],
        }), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


# The workload both arms report (the driver compares the two config objects).
CONFIG = {"workload": WORKLOAD,
          "inputs": "600 MB of fields per projection resident on the device (> 126 MB L2); "
                    "every step projects the same input velocities",
          "tolerance": "||b - A p||_2 <= 1e-6 ||b||_2, FP64 residual of the returned pressure"}
REF_PCG_SAMPLE_ITERS = 10  # PCG iterations per step of the reference arm's bounded sample


def reference_arm(args):
    """--impl reference: the reference's projection algorithm (divergence,
    Jacobi-PCG to its own stopping rule at tol 1e-6, gradient subtract,
    diagnostic divergence; fluid.py:612-734 with pressure_solve_pcg.cu:
    89-243) restated in C (oracle/, OpenMP on every host thread) on the same
    384x384x256 workload.  A full projection needs REF_PCG_ITERS_FALLBACK PCG
    iterations (about 80 s on the CPU), so each step is a bounded sample:
    REF_PCG_SAMPLE_ITERS PCG iterations from the cold start on the full grid.
    ms_per_step is that sample's measured time; value extrapolates it to
    projections/s = 1 / (t_setup + N t_iter + 2 t_div + t_grad) with t_iter
    from the timed steps (setup subtracted) and N the iteration count of the
    reference's stopping rule on this workload."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O

    mat, ux, uy, uz = _workload()
    threads = os.cpu_count() or 1
    O.set_threads(threads)
    J = REF_PCG_SAMPLE_ITERS

    def timed(fn):
        t0 = time.perf_counter()
        r = fn()
        return r, time.perf_counter() - t0

    div, t_div = timed(lambda: O.divergence(ux, uy, uz, mat, DX))
    p0 = np.zeros(mat.shape, np.float32)
    _, t_grad = timed(lambda: O.subtract_gradient(ux, uy, uz, p0, mat, DX, DT, RHO))
    t_setup = float(np.median([timed(lambda: O.pcg(div, mat, DX, DT, RHO, 1e-30, 0))[1]
                               for _ in range(3)]))
    for _ in range(args.warmup):
        O.pcg(div, mat, DX, DT, RHO, 1e-30, J)
    steps = []
    for _ in range(args.steps):
        steps.append(timed(lambda: O.pcg(div, mat, DX, DT, RHO, 1e-30, J))[1])
    t_step = float(np.mean(steps))
    t_iter = max(t_step - t_setup, 1e-9) / J
    n_ref = REF_PCG_ITERS_FALLBACK
    t_proj = t_setup + n_ref * t_iter + 2 * t_div + t_grad
    value = 1.0 / t_proj
    sample = (f"{J} PCG iterations from the cold start on the full 384x384x256 grid per step "
              f"({t_step * 1e3:.0f} ms; setup {t_setup * 1e3:.0f} ms, {t_iter * 1e3:.1f} "
              f"ms/iteration); value extrapolated to the {n_ref} iterations the reference's "
              f"stopping rule needs here (measured on the GPU with the reference-compatible "
              f"pressure_solve_pcg_launch) plus divergence x2 and gradient once")
    line = {"metric": METRIC, "value": value, "unit": "projections/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_step * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "fp32 arithmetic, fp64 dot products", "data": "synthetic",
            "impl": "reference", "config": dict(CONFIG, parallelism=f"replicas x{args.gpus}"),
            "method": "Jacobi-preconditioned CG (the reference's pressure_solve_pcg algorithm) "
                      "restated in C, OpenMP",
            "value_basis": "extrapolated: ms_per_step is the measured bounded sample; value = "
                           "1 / (t_setup + N t_iter + 2 t_div + t_grad)",
            "reference_iterations_to_tol": n_ref,
            "cpu_baseline": {"value": value, "unit": "projections/s", "cores": threads,
                             "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": "projections/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_projection(args, dev, rank, world, local, dist):
    """The headline: projections/s to FP64 rel-residual 1e-6 at 384x384x256.

    value: learned + mixed -- the network's pressure (tensor-core inference,
    boilingsim_b200.learned.WarmStart) starts the FP16-stored multigrid-CG
    solve inside every timed step.  Beside it, each measured the same way:
    mixed alone (cold start), the same solver with FP32 storage, and the plain
    FP32 Jacobi drop-in to the same tolerance (extrapolated, see
    plain_fp32_to_tolerance)."""
    import ctypes

    import torch

    from boilingsim_b200 import _lib
    from boilingsim_b200 import fluid as F
    from boilingsim_b200 import learned as LR
    from boilingsim_b200.solver import TolSolver

    mat, ux, uy, uz = _workload()
    nx, ny, nz = mat.shape
    n = mat.size
    mat_t = torch.as_tensor(mat).to(dev)
    mask = F.cell_mask(mat_t)
    u0 = [torch.as_tensor(a).to(dev) for a in (ux, uy, uz)]
    u = [a.clone() for a in u0]
    p = torch.zeros(mat.shape, dtype=torch.float32, device=dev)
    div = torch.zeros_like(p)
    max_div = torch.zeros(1, dtype=torch.float32, device=dev)
    solvers = {"fp16": TolSolver(mask, "fp16", device=dev),
               "fp32": TolSolver(mask, "fp32", device=dev)}
    net = LR.UNet.load(device=dev)
    warm = LR.WarmStart(net, mat_t, mask, mode=args.warm_mode)
    stream = torch.cuda.current_stream()
    last = {}

    # Timed steps project their own resident copy of the input velocities
    # (one per step, refreshed from u0 before the timed region), so no
    # restore copy runs inside it; above POOL_MAX steps, and in untimed
    # steps, the input is restored into u at the start of the step.
    POOL_MAX = 32
    pool = []

    def step(kind, graph=not args.host_driven, uu=None):
        if uu is None:
            for a, b in zip(u, u0):
                a.copy_(b, non_blocking=True)
            uu = u
        F.compute_divergence(div, *uu, mask, DX)
        if kind == "learned":
            warm.guess(div, DX, DT, RHO, out=p, graph=graph)
            res = solvers["fp16"].solve(div, DX, DT, RHO, tol=TOL, p=p, warm_start=True,
                                        graph=graph, want_x64=False)
        else:
            res = solvers["fp32" if kind == "fp32" else "fp16"].solve(div, DX, DT, RHO, tol=TOL,
                                                                      p=p, graph=graph,
                                                                      want_x64=False)
        F.subtract_pressure_gradient(*uu, p, mask, DX, DT, RHO)
        F.compute_divergence(div, *uu, mask, DX, max_div)
        last[kind] = res

    ncls = 12
    prof_ms = (ctypes.c_double * ncls)()
    prof_n = (ctypes.c_longlong * ncls)()
    peak, peak_kind = _peaks()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def time_steps(kind, k):
        staged = k <= POOL_MAX
        if staged:
            while len(pool) < k:
                pool.append([a.clone() for a in u0])
            for f in pool[:k]:
                for a, b in zip(f, u0):
                    a.copy_(b, non_blocking=True)
        torch.cuda.synchronize()
        ev0.record(stream)
        for i in range(k):
            step(kind, uu=pool[i] if staged else None)
        ev1.record(stream)
        torch.cuda.synchronize()
        return ev0.elapsed_time(ev1) / k

    def sweep_bytes():
        """Bytes one ZNF sweep moves: 13 per cell (p, rhs, mask in; p out) in the
        128-cell k row segments that hold a fluid cell, 9 (mask and p of the
        next plane in, +0 out) in the segments without one, which read
        neither rhs nor their j neighbours."""
        fl = (mask & 0x80) != 0
        pad = (-nz) % 128
        if pad:
            fl = torch.nn.functional.pad(fl.to(torch.uint8), (0, pad)).bool()
        seg = fl.reshape(nx, ny, -1, 128).any(dim=-1)
        cells_fluid_seg = int(seg.sum().item()) * 128
        cells_fluid_seg = min(cells_fluid_seg, n)
        return 13 * cells_fluid_seg + 9 * (n - cells_fluid_seg), cells_fluid_seg

    def plain_sweep():
        """200 sweeps of the reference-contract FP32 Jacobi kernel, event-timed:
        one sweep per HBM pass (tblock 1; its roofline on the bytes it moves,
        sweep_bytes), and pairs of sweeps per pass (temporal blocking, tblock 2;
        effective bandwidth = 13 B/cell per sweep / time per sweep)."""
        rhs = torch.empty_like(p)
        q = torch.empty_like(p)
        F.compute_divergence(div, *u0, mask, DX)
        sb, cells_fl = sweep_bytes()
        out = {}
        for tb in (1, 2):
            p.zero_()
            _lib.call("bsp_profile_enable", 1)
            _lib.lib().bsp_profile_read(None, None, 0)
            _lib.call("bsp_jacobi_solve", _lib.ptr(p), _lib.ptr(q), _lib.ptr(div),
                      _lib.ptr(rhs), _lib.ptr(mask), nx, ny, nz, DX, DT, RHO, 200, tb,
                      _lib.stream_handle())
            torch.cuda.synchronize()
            _lib.call("bsp_profile_enable", 0)
            _lib.lib().bsp_profile_read(prof_ms, prof_n, ncls)
            sweep_ms = prof_ms[0] / 200.0
            gbs = (sb if tb == 1 else 13.0 * n) / (sweep_ms * 1e-3) / 1e9
            out[tb] = {"ms_per_sweep": round(sweep_ms, 5), "GB/s": round(gbs, 1),
                       "frac": round(gbs / peak, 4), "launches": int(prof_n[0])}
        one = out[1]
        return {"ms": one["ms_per_sweep"], "GB/s": one["GB/s"], "frac": one["frac"],
                "bytes_per_sweep": sb,
                "bytes_rule": "13 B/cell in 128-cell k row segments holding a fluid cell "
                              f"({cells_fl} cells), 9 B/cell in the others (no rhs or j "
                              "neighbours read there)",
                "reference_contract_bytes_per_cell": 13,
                "GB/s_at_13B_per_cell": round(13.0 * n / (one["ms_per_sweep"] * 1e-3) / 1e9, 1),
                "temporal_blocking_2": {"ms_per_sweep": out[2]["ms_per_sweep"],
                                        "effective_GB/s": out[2]["GB/s"],
                                        "effective_frac": out[2]["frac"],
                                        "passes": out[2]["launches"]}}

    if args.only_sweep or args.only_conduction or args.only_advection:
        if rank == 0 and args.only_sweep:
            print(json.dumps({"plain_fp32_jacobi_sweep": plain_sweep()}), flush=True)
        if rank == 0 and args.only_conduction:
            print(json.dumps({"conduction": conduction_bench(mat, dev, *_peaks(), cpu=False)}),
                  flush=True)
        if rank == 0 and args.only_advection:
            print(json.dumps({"advection": advection_bench(mat, ux, uy, uz, dev, *_peaks(),
                                                           cpu=False)}), flush=True)
        if dist:
            dist.destroy_process_group()
        return

    kind = args.method
    for k in ("learned", "mixed", "fp32"):
        for _ in range(args.warmup if k == kind else (0 if args.skip_extras else 2)):
            step(k)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    clocks = Clocks(local)
    ms = time_steps(kind, args.steps)
    clk = clocks.stop()
    ms = max_over_ranks(ms, dist, dev)
    res = last[kind]
    others = {}
    if not args.skip_extras:
        for k in ("learned", "mixed", "fp32"):
            if k == kind:
                continue
            kk = max(3, min(args.steps, 10))
            others[k] = {"ms_per_step": round(time_steps(k, kk), 4), "steps": kk,
                         "inner_iterations": last[k].inner_iterations,
                         "outer_iterations": last[k].outer_iterations,
                         "rel_residual_fp64": last[k].rel_residual}
    # Per-kernel-class breakdown: the same step again with the library's event
    # timing on -- a second, host-driven pass (two events around every launch;
    # graphs suspend the event timing), so its total differs from ms_per_step.
    _lib.call("bsp_profile_enable", 1)
    _lib.lib().bsp_profile_read(None, None, 0)  # clear
    for _ in range(args.steps):
        step(kind, graph=False)
    torch.cuda.synchronize()
    _lib.call("bsp_profile_enable", 0)
    _lib.lib().bsp_profile_read(prof_ms, prof_n, ncls)
    if dist:
        dist.barrier()

    # ---- roofline of the dominant kernel class -------------------------------------
    # Algorithmic bytes per launch = bytes per cell x the cells the kernel
    # processes.  The level-0 column kernels (restriction, prolongation, A.ps,
    # CG update, FP64 residual) skip CTA tiles holding no fluid cell, so they
    # process n_act = the cells of the tiles with fluid; the x update is flat.
    nsm = torch.cuda.get_device_properties(dev).multi_processor_count
    n_act = active_tile_cells(mat, nsm)
    ts = 4 if kind == "fp32" else 2
    per_launch = {0: 13.0 * n,
                  1: (ts + 1 + ts / 8) * n_act,                # r, mask -> r_coarse
                  2: (ts + 1 + ts / 8 + ts) * n_act,           # r, mask, e_coarse -> z
                  3: (2 * ts + 1 + 2 * ts) * n_act,            # z, ps_prev, mask -> ps, Ap
                  4: (4 + 3 * ts + 4 + ts) * n_act,            # e, ps, Ap, r -> e, r
                  5: (13 + (ts + 4) / 2) * n_act,              # mask, x, div; rhat, e (write pass)
                  6: 20.0 * n}                                 # x, e -> x
    if prof_n[4] == 0:
        # CG update fused into the restriction: r_in, Ap, mask, e, ps -> r_out, e, r_coarse
        per_launch[1] = (4 * ts + 9 + ts / 8) * n_act
    names = {0: "jacobi_sweep",
             1: "mg_restrict_fine" if prof_n[4] else "cg_update_restrict_fine",
             2: "mg_prolong_smooth_fine", 3: "cg_direction_Ap", 4: "cg_update",
             5: "residual_fp64", 6: "x_update_fp64", 7: "mg_coarse_levels",
             8: "control_and_setup", 9: "divergence_gradient", 10: "learned_warm_start",
             11: "mg_levels_1_2_tiles"}
    total_ms = sum(prof_ms[c] for c in range(ncls)) or 1.0
    top = max((c for c in range(ncls) if prof_n[c] > 0), key=lambda c: prof_ms[c])
    dom = max((c for c in per_launch if prof_n[c] > 0), key=lambda c: prof_ms[c])
    avg_ms = prof_ms[dom] / prof_n[dom]
    bytes_launch = per_launch[dom]
    achieved = bytes_launch / (avg_ms * 1e-3) / 1e9
    traffic = CAPTURED_TRAFFIC.get((names[dom], "fp16" if ts == 2 else "fp32")) if (
        nx, ny, nz) == (384, 384, 256) else None
    roofline = {"bound": "hbm", "kernel": names[dom], "achieved": round(achieved, 1),
                "peak": peak, "unit": "GB/s", "frac": round(achieved / peak, 4),
                "traffic": traffic, "traffic_source": "ncu capture, one launch" if traffic
                else None, "peak_source": peak_kind,
                "algorithmic_bytes_per_launch": round(bytes_launch),
                "cells_processed_per_launch": int(n if dom in (0, 6) else n_act),
                "avg_launch_ms": round(avg_ms, 5),
                "share_of_step": round(prof_ms[dom] / total_ms, 3),
                "note": "the dominant HBM-bound class; the largest class overall is "
                        "'largest_class'"}
    largest = {"kernel": names[top], "share_of_step": round(prof_ms[top] / total_ms, 3),
               "ms_per_step": round(prof_ms[top] / args.steps, 4),
               "launches_per_step": prof_n[top] / args.steps}
    if top == 11:
        cycles = prof_n[2] / args.steps
        largest.update({"bound": "latency (eight tile-kernel launches per V-cycle on levels "
                                 "1-3, L2-resident: two smoothing sweeps a side on level 1)",
                        "us_per_cycle": round(1e3 * prof_ms[11] / max(prof_n[2], 1), 2),
                        "cycles_per_step": cycles})
    if top == 7:
        # one level-0 prolongation per V-cycle and one cooperative launch for
        # the levels below the tile-kernel ones
        cycles = prof_n[2] / args.steps
        largest.update({"bound": "latency (the phases of one cluster launch per V-cycle)",
                        "us_per_cycle": round(1e3 * prof_ms[7] / max(prof_n[2], 1), 2),
                        "cycles_per_step": cycles})
    kernel_ms = {names[c]: round(prof_ms[c] / args.steps, 4) for c in range(ncls) if prof_n[c]}
    kernel_gbs = {names[c]: round(per_launch[c] / (prof_ms[c] / prof_n[c] * 1e-3) / 1e9, 1)
                  for c in per_launch if prof_n[c]}
    launches = int(sum(prof_n))  # every kernel launch of the timed steps is instrumented

    sweep = e2e = cond = adv = plain = refcuda = None
    ref_iters = args.ref_iters or REF_PCG_ITERS_FALLBACK
    cpu = None
    if not args.skip_extras:
        sweep = plain_sweep()
        F.compute_divergence(div, *u0, mask, DX)
        plain = plain_fp32_to_tolerance(mat_t, mask, div, solvers["fp32"], dev,
                                        sweeps=args.plain_sweeps)
        t_dg = kernel_ms.get("divergence_gradient", 0.0)
        plain["ms_per_projection_extrapolated"] = round(
            plain["sweeps_to_tol_extrapolated"] * plain["ms_per_sweep"] + t_dg, 1)
        plain["projections_per_s_extrapolated"] = 1e3 / plain["ms_per_projection_extrapolated"]
        # the reference-compatible PCG (this library's kernels): iterations to
        # the reference's own stopping rule, and its time
        from boilingsim_b200.sim_core import SimCore, pcg_workspace

        F.compute_divergence(div, *u0, mask, DX)
        w = pcg_workspace(mat.shape, dev)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ref_iters_meas = SimCore(local).pressure_solve_pcg(
            _lib.ptr(p), _lib.ptr(div), _lib.ptr(mat_t), nx, ny, nz, DX, DT, RHO, TOL, 20000,
            *[_lib.ptr(w[k]) for k in ("b", "r", "z", "p_search", "Ap", "dot_ws", "alpha",
                                        "beta", "rzold", "rznew", "bsq", "rsq", "pAp")])
        torch.cuda.synchronize()
        ours_pcg_ms = (time.perf_counter() - t0) * 1e3
        if not args.ref_iters:
            ref_iters = ref_iters_meas
        refcuda = reference_cuda_block(
            mat_t, div, dev, sweep["ms"],
            {"ours_same_algorithm_ms": round(ours_pcg_ms, 2), "ours_iterations": ref_iters_meas,
             "ours_tolerance_solve_ms": round(others.get("mixed", {}).get("ms_per_step", ms), 3),
             "ours_tolerance_solve_note": "mixed (FP16-stored multigrid CG, FP64 refinement) "
                                          "full projection step, true FP64 residual <= 1e-6"})
        if "pcg_to_1e-6" in refcuda:
            r = refcuda["pcg_to_1e-6"]
            r["speedup_same_algorithm"] = round(r["reference_ms"] / ours_pcg_ms, 2)
            r["speedup_tolerance_solve"] = round(r["reference_ms"] / r["ours_tolerance_solve_ms"],
                                                 2)
        cond = conduction_bench(mat, dev, peak, peak_kind,
                                cpu=rank == 0 and world == 1 and not args.no_cpu_baseline)
        adv = advection_bench(mat, ux, uy, uz, dev, peak, peak_kind,
                              cpu=rank == 0 and world == 1 and not args.no_cpu_baseline)

        # ---- end to end through the public API with host buffers ----------------------
        host_u = [torch.as_tensor(a).pin_memory() for a in (ux, uy, uz)]
        host_out = [torch.empty(a.shape, dtype=torch.float32).pin_memory() for a in (ux, uy, uz)]
        host_p = torch.empty(mat.shape, dtype=torch.float32).pin_memory()
        grid = F.Grid(nx, ny, nz, DX, p, mat_t, *u, mask=mask)
        ws = F.FluidWorkspace(div, torch.empty_like(p), max_div)
        cfg = F.ScenarioConfig(F.SolverConfig(pressure_tol=TOL))
        os.environ["BOILINGSIM_PRESSURE_SOLVER"] = {"learned": "b200-learned",
                                                    "mixed": "b200-mixed",
                                                    "fp32": "b200-mg"}[kind]
        F._TOL_SOLVERS.clear()
        F._TOL_SOLVERS[(id(grid), grid.shape, "fp16" if kind != "fp32" else "fp32")] = \
            solvers["fp32" if kind == "fp32" else "fp16"]
        F._WARM_STARTS[(id(grid), grid.shape)] = warm

        def e2e_step():
            for d, h in zip(u, host_u):
                d.copy_(h, non_blocking=True)
            md = F.pressure_projection(grid, ws, cfg, DT, RHO)
            host_p.copy_(p, non_blocking=True)
            for h, d in zip(host_out, u):
                h.copy_(d, non_blocking=True)
            torch.cuda.synchronize()
            return md

        e2e_step()
        e2e_steps = max(2, min(args.steps, 5))
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(e2e_steps):
            e2e_step()
        e2e_s = (time.perf_counter() - t0) / e2e_steps
        h2d = sum(a.numel() * 4 for a in host_u)
        d2h = sum(a.numel() * 4 for a in host_out) + host_p.numel() * 4 + 4
        # the same projections through fluid.ProjectionPipeline: three in
        # flight (measured: 54 projections/s with two, 70 with three, 70 with
        # four), each with its own device state and stream, so the copy
        # engines move one projection's fields while another computes
        depth = 3
        pipe = F.ProjectionPipeline(mat_t, DX, cfg, depth=depth)
        outs = [[torch.empty(a.shape, dtype=torch.float32).pin_memory() for a in (ux, uy, uz)] +
                [torch.empty(mat.shape, dtype=torch.float32).pin_memory()]
                for _ in range(depth)]

        def run_pipe(k):
            tickets, md = [], 0.0
            for q in range(k):
                if q >= depth:
                    md = pipe.result(tickets[q - depth])  # before its host buffers are reused
                tickets.append(pipe.submit(*host_u, *outs[q % depth], DT, RHO))
            for t in tickets[-depth:]:
                md = pipe.result(t)
            return md

        run_pipe(depth)  # graphs and plans of every slot
        pipe_steps = max(6, min(2 * args.steps, 12))
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        run_pipe(pipe_steps)
        pipe_s = (time.perf_counter() - t0) / pipe_steps
        # replicas: the slowest rank's host-timed rate, times the ranks
        pipe_ms = max_over_ranks(pipe_s * 1e3, dist, dev) if world > 1 else pipe_s * 1e3
        same = all(torch.equal(a, b) for a, b in zip(outs[(pipe_steps - 1) % depth],
                                                     host_out + [host_p]))
        del pipe
        e2e = {"value": round(job_rate(world, 1, pipe_ms), 3), "unit": "projections/s",
               "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
               "mode": "fluid.ProjectionPipeline, three projections in flight: per step the "
                       "pinned-host copy of u in, the projection, and u, p and max|div| "
                       "copied out, timed on the host clock over the steps",
               "steps": pipe_steps, "same_result_as_sequential": bool(same),
               "sequential": {"value": round(1.0 / e2e_s, 3),
                              "mode": "fluid.pressure_projection one at a time"}}

        if rank == 0 and world == 1 and not args.no_cpu_baseline:
            cpu = cpu_reference(mat, ux, uy, uz, ref_iters)
            cpu = {k: cpu[k] for k in ("value", "unit", "cores", "kind", "sample")}

    if rank == 0:
        value = job_rate(world, 1, ms)
        ratio = None
        if plain:
            ratio = {"learned_mixed_over_plain_fp32": round(
                value / plain["projections_per_s_extrapolated"], 1) if kind == "learned" else
                None, "target": 4.0}
            for k, v in others.items():
                ratio[f"{k}_over_plain_fp32"] = round(
                    1e3 / v["ms_per_step"] / plain["projections_per_s_extrapolated"], 1)
            if kind == "learned" and "mixed" in others:
                ratio["learned_mixed_over_mixed"] = round(others["mixed"]["ms_per_step"] / ms, 3)
        method = {"learned": "learned warm start (U-Net on tcgen05 tensor cores, "
                             f"{warm.mode} resolution) + FP16-stored multigrid-CG, FP64 "
                             "iterative refinement",
                  "mixed": "FP16-stored multigrid-CG, FP64 iterative refinement (cold start)",
                  "fp32": "FP32-stored multigrid-CG, FP64 iterative refinement (cold start)"}
        line = {
            "metric": METRIC, "value": round(value, 3), "unit": "projections/s",
            "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(ms, 4), "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None,
            "dtype": ("fp16 storage / fp32 arithmetic / fp64 residual and dot products; "
                      "bf16 network" if kind != "fp32" else
                      "fp32 storage and arithmetic / fp64 residual and dot products"),
            "data": "synthetic",
            "config": dict(CONFIG, parallelism=f"replicas x{world}"),
            "method": {"name": kind, "description": method[kind],
                       "launch": ("host-driven refinement loop" if args.host_driven else
                                  "one device-driven CUDA graph per solve"),
                       "input_staging": (
                           "each timed step projects its own resident copy of the input "
                           "velocities (454 MB), staged before the timed region"
                           if args.steps <= POOL_MAX else
                           "the input velocities are restored at the start of every step")},
            "guess": ({"mode": warm.mode, "keep_below": warm.keep_below,
                       "rel_residual_of_scaled_guess": round(float(warm.relres.item()), 4),
                       "gamma": float(warm.gamma.item()),
                       "kept": float(warm.gamma.item()) != 0.0,
                       "rule": "the energy-scaled guess starts the solve only when its "
                               "relative residual is below keep_below, else the solve "
                               "starts from zero (decided on the device; the network's time "
                               "stays in the step)"} if kind == "learned" else None),
            "solve": {"inner_iterations": res.inner_iterations,
                      "outer_iterations": res.outer_iterations, "levels": res.levels,
                      "rel_residual_fp64": res.rel_residual, "status": res.status},
            "others": others,
            "plain_fp32_jacobi_to_tol": plain,
            "ratios": ratio,
            "kernel_ms_per_step_host_driven_pass": kernel_ms,
            "kernel_algorithmic_GBs": kernel_gbs,
            "largest_class": largest,
            "roofline": roofline,
            "plain_fp32_jacobi_sweep": sweep,
            "reference_cuda": refcuda,
            "conduction": cond,
            "advection": adv,
            "reference_pcg_iterations_to_tol": ref_iters,
            "cpu_baseline": cpu,
            "e2e": e2e,
            "gpu_launches": launches,
            "clocks": clk,
        }
        print(json.dumps(line), flush=True)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    # FP16 storage of the inner iterates (FP32 arithmetic, FP64 residual and
    # reductions) is the mixed-precision method the metric names; fp32 is the
    # same solver with FP32 storage
    ap.add_argument("--storage", default="fp16", choices=["fp32", "fp16", "bf16"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--host-driven", action="store_true",
                    help="drive the refinement loop from the host instead of running each "
                         "solve as one device-driven CUDA graph")
    ap.add_argument("--ref-iters", type=int, default=0,
                    help="reference PCG iteration count to use instead of measuring it")
    ap.add_argument("--skip-extras", action="store_true",
                    help="timed projections only (no sweep, e2e, reference iterations or CPU "
                         "baseline): the short form used under ncu")
    ap.add_argument("--only-sweep", action="store_true",
                    help="run only the plain FP32 Jacobi sweep measurement (for ncu)")
    ap.add_argument("--only-conduction", action="store_true",
                    help="run only the backward-Euler conduction measurement (for ncu)")
    ap.add_argument("--only-advection", action="store_true",
                    help="run only the semi-Lagrangian advection measurement (for ncu)")
    ap.add_argument("--method", default="learned", choices=["learned", "mixed", "fp32"],
                    help="the timed step: learned warm start + FP16-stored solve (the metric's "
                         "learned+mixed), the FP16-stored solve alone, or FP32 storage")
    ap.add_argument("--warm-mode", default="auto", choices=["auto", "full", "coarse", "coarse4"],
                    help="resolution of the network in the learned step")
    ap.add_argument("--plain-sweeps", type=int, default=8000,
                    help="plain FP32 Jacobi sweeps measured before extrapolating to tolerance")
    ap.add_argument("--config", default="projection",
                    choices=["projection", "batched", "learned"],
                    help="projection: the headline 384x384x256 projection; batched: 64 uneven "
                         "pot scenes (48^3 .. 128x128x96) solved in cooperative launches; learned: "
                         "the U-Net warm start on the 192x192x128 pots (walls 2/3/4)")
    args = ap.parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        if rank == 0:
            reference_arm(args)
        return

    import torch

    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
    dev = torch.device("cuda", local)
    if args.config == "batched":
        run_batched(args, dev, rank, world, dist)
        return
    if args.config == "learned":
        run_learned(args, dev, rank, world, dist)
        return
    run_projection(args, dev, rank, world, local, dist)


if __name__ == "__main__":
    main()
