#!/usr/bin/env python3
"""Benchmark: DOF/s to a 1e-8 relative residual on one GB300, mixed precision vs plain FP64.

Workload (the single-GPU configuration the metric is quoted on): Poisson -div(k grad u) = 1
on the unit cube, 128^3 hexahedra, Q2 Lagrangian elements, 3x3x3 Gauss points, interior
vertices perturbed by a seeded U(-0.15h, 0.15h) per component (trilinear geometry),
k = exp(N(0,1)) per cell, homogeneous Dirichlet on the whole boundary, Jacobi-PCG from
x0 = 0 to ||r|| <= 1e-8 ||r0||.  16,581,375 free dofs.

A step = numeric assembly (integration + CSR + FP32 copy + Jacobi diagonal) + PCG solve;
the symbolic phase (dof numbering, sparsity) is built once before timing ("warm" DOF/s).
value = free dofs / device time of a step (inputs resident in HBM), mixed precision
(FP32 matrix/SpMV/Jacobi inner PCG, dots in compensated FP32 and FP64, FP64 residual and refinement).  The plain FP64
drop-in is timed beside it.  e2e = the same through the public API with host buffers:
per-cell coefficients copied in from pinned host memory and the solution copied out.

--impl reference times the reference's CPU path (the C++ restatement in oracle/, the
reference itself is Fortran and cannot be built here) on all host cores: one complete solve
of the full workload.  The GPU arm's cpu_baseline is the same full-size oracle run, continued
to rtol 1e-13 to give the oracle solution the GPU solutions are compared with
(error_vs_oracle).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

SEED = 20261203
METRIC = "DOF/s to 1e-8 rel. residual, mixed vs plain FP64 on GB300; p50/p99 solve latency"


def workload(n, seed=SEED):
    rng = np.random.Generator(np.random.PCG64(seed))
    h = 1.0 / n
    nv = n + 1
    k, j, i = np.meshgrid(np.arange(nv), np.arange(nv), np.arange(nv), indexing="ij")
    xyz = np.stack([i * h, j * h, k * h], axis=-1).reshape(-1, 3)
    ii, jj, kk = i.ravel(), j.ravel(), k.ravel()
    interior = (ii > 0) & (ii < n) & (jj > 0) & (jj < n) & (kk > 0) & (kk < n)
    d = rng.uniform(-0.15 * h, 0.15 * h, size=xyz.shape)
    xyz[interior] += d[interior]
    coef = np.exp(rng.normal(0.0, 1.0, size=n ** 3))
    return np.ascontiguousarray(xyz.ravel()), coef


def spmv_bytes(n, nnz, fp32):
    """Algorithmic HBM bytes of one SpMV: every nonzero value read once, x read once, y written
    once (no index bytes: the lattice-implicit layout stores none)."""
    return (4 * nnz + 8 * n) if fp32 else (8 * nnz + 16 * n)


def csr_bytes(n, nnz, fp32):
    """The same for a full CSR matrix with int32 columns (the explicit-index reference figure)."""
    return (8 * nnz + 4 * (n + 1) + 8 * n) if fp32 else (12 * nnz + 4 * (n + 1) + 16 * n)


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in self.lines:
            p = [x.strip() for x in l.split(",")]
            if len(p) < 9:
                continue
            try:
                sm.append(float(p[1]))
                smax.append(float(p[2]))
            except ValueError:
                continue
            for nm, v in zip(names, p[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        loaded = [s for s in sm if s > 0.5 * max(sm)] or sm
        return {"sm_mhz": statistics.median(loaded), "sm_max_mhz": max(smax), "reasons": sorted(reasons),
                "samples": len(sm)}


def peaks():
    try:
        return json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        return None


def host_threads():
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def workload_config(n, nfree, nnz_full, nnz_upper):
    """The workload's description; both arms print exactly this dict (no run-dependent values)."""
    b32, b64 = spmv_bytes(nfree, nnz_full, True), csr_bytes(nfree, nnz_full, False)
    return {"workload": f"poisson_q2_{n}^3_perturbed_lognormal_jacobi_pcg_1e-8", "n": n, "order": 2,
            "num_free_dofs": nfree, "nnz_full": nnz_full, "nnz_upper": nnz_upper, "precond": "jacobi",
            "rtol": 1e-8, "criterion": "res_res, x0 = 0", "geometry": "interior vertices U(+-0.15h), trilinear",
            "coefficient": "k = exp(N(0,1)) per cell", "source": "f = 1", "dirichlet": "u = 0 on the whole boundary",
            "seed": SEED,
            "l2": "inputs larger than L2 (FP32 matrix %.1f GB, FP64 CSR %.1f GB)" % (b32 / 1e9, b64 / 1e9)}


def oracle_solve(n, nthreads, rtol, kernel="sym", maxit=200000, seed=SEED):
    """The oracle (C++ restatement of the reference's serial path) on the full workload: mesh and
    dof numbering, numeric assembly (element integration, COO append, sort_and_compress) and
    Jacobi-PCG from x0 = 0, on `nthreads` host threads.  The CSR is bit-identical to the
    serial restatement's; the threaded SpMV (the symmetric-storage kernel, or "gather": a full
    CSR row gather) sums in another order, so iterates agree with the serial ones to rounding.
    Returns the problem, the solve record and stage times (s)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    O.build()
    xyz, coef = workload(n, seed)
    P = O.Problem([n, n, n], order=2, vertex_xyz=xyz, cell_coef=coef, source_fn=O.FN_CONST, fn_param=[1.0],
                  nthreads=nthreads)
    tm = P.timings()
    nth = -nthreads if (kernel == "gather" and nthreads > 1) else nthreads
    r = P.cg(precond=1, rtol=rtol, maxit=maxit, nthreads=nth, times=True, history=True)
    bnorm = float(np.linalg.norm(P.rhs()))
    return P, r, {"setup": float(tm["setup"]), "integrate": float(tm["integrate"]),
                  "compress": float(tm["compress"]), "bnorm": bnorm}


def time_to_rtol(r, bnorm, rtol):
    """(iterations, seconds) at which the res_res test ||r_k|| <= rtol ||b|| first held, read off
    a longer run's history (CG's iterates do not depend on its stopping test)."""
    h = r["history"]
    hit = np.nonzero(h <= rtol * bnorm)[0]
    if hit.size == 0:
        return None, None
    k = int(hit[0])
    return k + 1, float(r["times"][k])


def cpu_baseline_full(n, nthreads, kernel, oracle_rtol):
    """CPU baseline on the FULL workload (no sample, no scaling): the oracle's numeric assembly
    plus Jacobi-PCG to rtol 1e-8, timed on `nthreads` host threads.  The PCG runs on to
    `oracle_rtol`; the 1e-8 time is read at the iteration where the residual test first held,
    and the solution at `oracle_rtol` is the oracle solution the GPU results are compared with."""
    P, r, tm = oracle_solve(n, nthreads, oracle_rtol, kernel)
    its8, t8 = time_to_rtol(r, tm["bnorm"], 1e-8)
    t_asm = tm["integrate"] + tm["compress"]
    rec = {"value": P.nfree / (t_asm + t8) if t8 else None, "unit": "DOF/s", "cores": nthreads, "kind": "port",
           "sample": f"the full workload ({n}^3 Q2, {P.nfree} dofs), not a sample: oracle numeric assembly "
                     f"({tm['integrate']:.2f} s integration + COO append, {tm['compress']:.2f} s sort_and_compress) + "
                     f"{its8} Jacobi-PCG iterations to 1e-8 ({t8:.2f} s, {kernel} SpMV) on {nthreads} threads; "
                     f"dof numbering ({tm['setup']:.2f} s) excluded as on the GPU",
           "assembly_s": t_asm, "pcg_s": t8, "iterations": its8, "setup_s": tm["setup"], "threads": nthreads,
           "spmv": kernel, "cpu": cpu_model()}
    return P, r, rec


def cpu_model():
    try:
        out = subprocess.run(["lscpu"], capture_output=True, text=True, timeout=10).stdout
        for line in out.splitlines():
            if line.startswith("Model name"):
                return line.split(":", 1)[1].strip()
    except Exception:
        pass
    return None


def run_reference(args):
    """The reference's CPU path (its C++ restatement: the reference is Fortran and no Fortran
    compiler exists here) on every host thread.  Warm-up: W complete solves of a smaller mesh
    of the same distribution.  Timed: ONE complete solve of the full workload (numeric assembly
    + Jacobi-PCG to 1e-8); the line reports it over the K requested steps, so that
    steps x ms_per_step is that solve's time."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    nth = host_threads()
    for _ in range(args.warmup):
        oracle_solve(args.ref_warm_n, nth, 1e-8, args.oracle_kernel)
    P, r, tm = oracle_solve(args.n, nth, 1e-8, args.oracle_kernel)
    t_asm = tm["integrate"] + tm["compress"]
    t_solve = t_asm + float(r["times"][-1])
    v = P.nfree / t_solve
    nnz_up = P.nnz_upper
    cfg = workload_config(args.n, P.nfree, 2 * nnz_up - P.nfree, nnz_up)
    ms = t_solve * 1e3 / max(1, args.steps)
    line = {"metric": METRIC, "value": v, "unit": "DOF/s", "impl": "reference", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": f"synthetic (PCG64 seed {SEED}): perturbed vertices U(+-0.15h), k=exp(N(0,1)) per cell, f=1",
            "config": cfg,
            "step_def": f"one complete solve of the workload is timed (numeric assembly {t_asm:.2f} s + "
                        f"{r['iters']} PCG iterations {float(r['times'][-1]):.2f} s = {t_solve:.2f} s) and divided "
                        f"over the {args.steps} steps: steps x ms_per_step = the solve time; warm-up = "
                        f"{args.warmup} complete solves at {args.ref_warm_n}^3",
            "solves_timed": 1, "solve_ms": t_solve * 1e3, "p50_ms": t_solve * 1e3, "p99_ms": t_solve * 1e3,
            "iterations": r["iters"], "converged": bool(r["converged"]),
            "assembly_ms": t_asm * 1e3, "pcg_ms": float(r["times"][-1]) * 1e3, "dof_numbering_ms": tm["setup"] * 1e3,
            "implementation": "reference path restated in C++ (oracle/fempar_oracle.cpp; the reference is Fortran, "
                              "no Fortran compiler on the image): COO append + sort_and_compress, upper-triangle CSR, "
                              f"CG with Jacobi; {nth} OpenMP threads, {args.oracle_kernel} SpMV",
            "cpu_baseline": {"value": v, "unit": "DOF/s", "cores": nth, "kind": "port",
                             "sample": f"the full workload ({args.n}^3), one complete solve on {nth} threads",
                             "cpu": cpu_model()},
            "e2e": {"value": v, "unit": "DOF/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


# DRAM bytes of one iteration of the FP32 CG kernel per byte it stores or updates (k_pcg32 at 64^3 Q2, one
# ncu capture of a 16-iteration launch: 9138 MB read + 444 MB written, against 16 x 635 MB of values and
# vectors): the vectors stay in L2 at that size
DRAM_PER_FORMAT_BYTE_PCG32 = 599.0 / 635.3


def replica_aggregate(dist, times_ms, units, device="cpu"):
    """Replicas (one independent problem per rank, no data-path collective): each timing
    becomes the maximum over the ranks and the work the sum of every rank's units, so a
    rate = units / max time.  dist = torch.distributed (initialised) or None for one rank."""
    import torch
    if dist is None:
        return list(times_ms), units
    t = torch.tensor(list(times_ms), dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    u = torch.tensor([float(units)], dtype=torch.float64, device=device)
    dist.all_reduce(u, op=dist.ReduceOp.SUM)
    return [float(v) for v in t.tolist()], float(u.item())


SHARP_WAVE = [50.0, 0.7, -0.05, -0.05, -0.05]


def plain_method_gpu(fg, ctx, stream, reps=5):
    """The reference's CPU-runnable case on the GPU, FP64 drop-in: Poisson on the unit cube,
    32^3 Q1, the sharp circular wave as Dirichlet data and source, unpreconditioned CG to 1e-8
    from x0 = 0.  DOF/s of numeric assembly + solve (CUDA events, median of `reps`)."""
    import torch
    tri = fg.SerialTriangulation(ctx, (32, 32, 32))
    sp = fg.SerialFESpace(tri, order=1, dirichlet_ids=fg.ALL_BOUNDARY_IDS)
    integ = fg.PoissonIntegration(source_fn=fg.FG_FN_SHARP_WAVE, boundary_fn=fg.FG_FN_SHARP_WAVE,
                                  fn_param=SHARP_WAVE)
    op = fg.FEAffineOperator(sp, integ).compute()
    s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "identity")
    s.set_parameters_from_pl({"ILS_RTOL": 1e-8, "ILS_MAX_NUM_ITERATIONS": 100000})
    x = torch.empty(sp.num_free_dofs, dtype=torch.float64, device=f"cuda:{ctx.device}")
    times = []
    for _ in range(reps + 2):
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        op.compute()
        s.solve_device(x=x)
        e1.record(stream)
        e1.synchronize()
        times.append(e0.elapsed_time(e1))
    ms = statistics.median(times[2:])
    out = {"workload": "poisson_q1_32^3_sharp_wave_cg_1e-8 (unpreconditioned, FP64 drop-in)",
           "num_free_dofs": sp.num_free_dofs, "value": sp.num_free_dofs / (ms * 1e-3), "unit": "DOF/s",
           "ms_per_solve": ms, "iterations": s.info()["iterations"], "x": x.cpu().numpy()}
    op.close()
    return out


def plain_method_cpu():
    """The same case on the oracle, serial (the reference's own single-threaded path): numeric
    assembly (integration, COO append, sort_and_compress) + CG, timed in full."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    O.build()
    P = O.Problem((32, 32, 32), order=1, source_fn=O.FN_SHARP_WAVE, boundary_fn=O.FN_SHARP_WAVE, fn_param=SHARP_WAVE)
    tm = P.timings()
    r = P.cg(precond=0, rtol=1e-8, maxit=100000, times=True)
    t = float(tm["integrate"]) + float(tm["compress"]) + float(r["times"][-1])
    return {"value": P.nfree / t, "unit": "DOF/s", "cores": 1, "kind": "port", "seconds": t,
            "iterations": r["iters"], "x": r["x"]}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--n", type=int, default=128)
    ap.add_argument("--fp64-steps", type=int, default=2)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--ref-warm-n", type=int, default=24)
    ap.add_argument("--oracle-kernel", default="sym", choices=["sym", "gather"])
    ap.add_argument("--oracle-rtol", type=float, default=1e-13)
    ap.add_argument("--no-extra", action="store_true", help="skip the 32^3 Q1 and batched-problem legs")
    ap.add_argument("--batch-count", type=int, default=4096)
    args = ap.parse_args()

    if args.impl == "reference":
        run_reference(args)
        return

    import torch
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device(f"cuda:{local}"))

    import fempar_gb300 as fg
    from fempar_gb300 import _lib as L
    import ctypes as C

    n = args.n
    xyz, coef = workload(n)
    ctx = fg.Context(local)
    sp_ptr = C.c_void_p()
    L.lib().fg_ctx_get_stream(ctx.h, C.byref(sp_ptr))
    stream = torch.cuda.ExternalStream(sp_ptr.value, device=f"cuda:{local}")

    t0 = time.perf_counter()
    tri = fg.SerialTriangulation(ctx, [n, n, n], vertex_xyz=xyz)
    space = fg.SerialFESpace(tri, order=2, dirichlet_ids=fg.ALL_BOUNDARY_IDS)
    t_symbolic = time.perf_counter() - t0
    coef_dev = torch.from_numpy(coef).to(f"cuda:{local}")
    integ_dev = fg.PoissonIntegration(cell_coef=coef_dev, source_fn=fg.FG_FN_CONST, fn_param=[1.0])
    # the mixed arm asks for fast integration (FG_FAST_INTEGRATION), the FP64 drop-in for FP64;
    # by default both get the tensor-core element matrices (FG_TC_INTEGRATION=2)
    integ_fast = fg.PoissonIntegration(cell_coef=coef_dev, source_fn=fg.FG_FN_CONST, fn_param=[1.0],
                                       fast_integration=True)
    op = fg.FEAffineOperator(space, integ_dev).compute()
    nfree = space.num_free_dofs
    nnz = space.info.nnz_full
    xbuf = torch.empty(nfree, dtype=torch.float64, device=f"cuda:{local}")

    def solver(precision):
        s = fg.IterativeLinearSolver().set_type_from_string("CG").set_operators(op, "jacobi")
        s.set_parameters_from_pl({"ILS_RTOL": 1e-8, "ILS_MAX_NUM_ITERATIONS": 200000,
                                  "PRECISION": "mixed" if precision == fg.FG_MIXED else "fp64"})
        return s

    def sync_all():
        torch.cuda.synchronize()
        if dist:
            dist.barrier()
            torch.cuda.synchronize()

    def timed_steps(precision, k, w, e2e=False, host=None):
        s = solver(precision)
        times, infos, launches = [], [], 0
        for it in range(w + k):
            sync_all()
            l0 = ctx.kernel_launches()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            if e2e:
                op.integration = host["integ"]
                op.compute()
                s.solve(out=host["x"])
            else:
                op.integration = integ_fast if precision == fg.FG_MIXED else integ_dev
                op.compute()
                s.solve_device(x=xbuf)
            e1.record(stream)
            e1.synchronize()
            if it >= w:
                times.append(e0.elapsed_time(e1))
                infos.append(s.info())
                launches += ctx.kernel_launches() - l0
        return times, infos, launches, s

    # ---- FP64 drop-in (reference algorithm) ----
    t64, i64, _, s64 = timed_steps(fg.FG_FP64, args.fp64_steps, 1)
    x64 = xbuf.clone()
    iters64 = i64[-1]["iterations"]
    # ---- mixed precision (headline) ----
    clk = ClockSampler(local)
    clk.start()
    tmx, imx, launches, smx = timed_steps(fg.FG_MIXED, args.steps, args.warmup)
    clocks = clk.stop()
    xmx = xbuf.clone()
    err_vs_fp64 = float(torch.linalg.norm(xmx - x64) / torch.linalg.norm(x64))
    # ---- end to end through the public API with pinned host buffers ----
    coef_pin = torch.from_numpy(coef).pin_memory()
    x_pin = torch.empty(nfree, dtype=torch.float64).pin_memory()
    host = {"integ": fg.PoissonIntegration(cell_coef=coef_pin.numpy(), source_fn=fg.FG_FN_CONST, fn_param=[1.0],
                                           fast_integration=True),
            "x": x_pin.numpy()}
    te2e, _, _, _ = timed_steps(fg.FG_MIXED, max(1, args.steps), 1, e2e=True, host=host)
    op.integration = integ_dev
    op.compute()

    # ---- dominant kernel: SpMV, timed on the library's stream ----
    def spmv_ms(precision, reps=20):
        # the solver's SpMV alone, back to back on the library's stream (matrix >> L2);
        # vectors in the solver layout (solver_vec_len entries)
        nvec = space.info.solver_vec_len
        if precision == fg.FG_MIXED:
            xv = torch.rand(nvec, dtype=torch.float32, device=f"cuda:{local}")
        else:
            xv = torch.rand(nvec, dtype=torch.float64, device=f"cuda:{local}")
        yv = torch.empty_like(xv)
        sync_all()
        op.apply_solver_layout_device(xv, yv, precision, reps=2)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        op.apply_solver_layout_device(xv, yv, precision, reps=reps)
        e1.record(stream)
        e1.synchronize()
        return e0.elapsed_time(e1) / reps

    def assembly_ms(integ, reps=3):
        op.integration = integ
        sync_all()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(reps):
            op.compute()
        e1.record(stream)
        e1.synchronize()
        return e0.elapsed_time(e1) / reps

    ms32 = spmv_ms(fg.FG_MIXED)
    ms64 = spmv_ms(fg.FG_FP64)
    ms_asm = assembly_ms(integ_fast)
    ms_asm64 = assembly_ms(integ_dev)
    op.integration = integ_dev
    op.compute()
    pk = peaks()
    hbm = pk["hbm_gbs"] if pk else 6800.0
    b32, b64 = spmv_bytes(nfree, nnz, True), spmv_bytes(nfree, nnz, False)
    ach32 = b32 / (ms32 * 1e-3) / 1e9
    ach64 = b64 / (ms64 * 1e-3) / 1e9
    nent, nvec = space.info.solver_entries, space.info.solver_vec_len
    layout = "lattice-implicit SELL-32x4 (no column indices)" if space.info.solver_layout == 0 else "SELL-32x4-256"
    kname = "k_stencil_spmv" if space.info.solver_layout == 0 else "k_sell_spmv"
    fmt32 = 4 * nent + 8 * nvec + (0 if space.info.solver_layout == 0 else 4 * nent)
    ms_it = imx[-1]["solve_ms"] / max(1, imx[-1]["iterations"])
    bit = 4 * nnz + 36 * nfree
    fmt_it = 4 * nent + 36 * nvec + (0 if space.info.solver_layout == 0 else 4 * nent)
    fmt64 = 8 * nent + 16 * nvec + (0 if space.info.solver_layout == 0 else 4 * nent)

    # ---- replicas: slowest rank's time, every rank's dofs ----
    dev = f"cuda:{local}"
    (ms_mx, ms_64, ms_e2e), total = replica_aggregate(
        dist, [statistics.mean(tmx), statistics.mean(t64), statistics.mean(te2e)], nfree, dev)
    value = total / (ms_mx * 1e-3)
    v64 = total / (ms_64 * 1e-3)
    ve2e = total / (ms_e2e * 1e-3)
    if rank != 0:
        if dist:
            dist.destroy_process_group()
        return
    # ---- the other configurations, after the timed region (rank 0, one GPU) ----
    cfg1, batch = None, None
    if not args.no_extra and world == 1:
        cfg1 = plain_method_gpu(fg, ctx, stream)
        from fempar_gb300.batch import benchmark as batch_benchmark
        batch = batch_benchmark(ctx, count=args.batch_count, runs=2, rtols=(1e-8, 1e-10), check=8)
    cb, oracle_err = None, None
    if cfg1 is not None and not args.no_cpu_baseline:
        c1 = plain_method_cpu()
        xg = cfg1.pop("x")
        cfg1["cpu_baseline"] = {k: v for k, v in c1.items() if k != "x"}
        cfg1["error_vs_oracle"] = float(np.linalg.norm(xg - c1["x"]) / np.linalg.norm(c1["x"]))
    elif cfg1 is not None:
        cfg1.pop("x")
    if not args.no_cpu_baseline and world == 1:
        try:
            P, r, cb = cpu_baseline_full(n, host_threads(), args.oracle_kernel, args.oracle_rtol)
            xo = r["x"]
            no = float(np.linalg.norm(xo))
            x64h, xmxh = x64.cpu().numpy(), xmx.cpu().numpy()
            oracle_err = {"fp64": float(np.linalg.norm(x64h - xo) / no), "mixed": float(np.linalg.norm(xmxh - xo) / no),
                          "oracle_rtol": args.oracle_rtol, "oracle_iterations": r["iters"],
                          "oracle_converged": bool(r["converged"]),
                          "def": "||x - x_oracle|| / ||x_oracle||, x_oracle = the oracle's Jacobi-PCG solution of the "
                                 "same workload (CPU, FP64) to the rtol above; x = the GPU solutions at rtol 1e-8"}
            del P
        except Exception as e:  # reported, never silently replaced
            cb = {"value": None, "unit": "DOF/s", "cores": host_threads(), "kind": "port", "sample": f"failed: {e}"}
    srt = sorted(tmx)
    line = {
        "metric": METRIC, "value": value, "unit": "DOF/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_mx, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "fp32 matrix/SpMV/Jacobi, dots in compensated fp32 and fp64, fp64 residual/refinement",
        "data": f"synthetic (PCG64 seed {SEED}): perturbed vertices U(+-0.15h), k=exp(N(0,1)) per cell, f=1",
        "config": workload_config(n, nfree, nnz, space.info.nnz_upper),
        "parallelism": "replicas" if world > 1 else "single", "symbolic_s": t_symbolic,
        "p50_ms": srt[len(srt) // 2], "p99_ms": srt[min(len(srt) - 1, int(round(0.99 * (len(srt) - 1))))],
        "iterations": imx[-1]["iterations"], "outer_iterations": imx[-1]["outer_iterations"],
        "assembly_ms": ms_asm, "assembly_fp64_ms": ms_asm64,
        "mixed_integration": "element matrices of both arms: one emulated-FP64 tensor-core product of the cells' "
                             "geometric factors with the shared reference-gradient table (FG_TC_INTEGRATION=2)",
        "solve_ms": imx[-1]["solve_ms"],
        "error_vs_fp64": err_vs_fp64,
        "error_vs_oracle": oracle_err,
        "fp64": {"value": v64, "ms_per_step": ms_64, "iterations": iters64, "dtype": "f64"},
        "mixed_vs_fp64": value / v64,
        "e2e": {"value": ve2e, "unit": "DOF/s", "h2d_bytes_per_step": int(coef.nbytes),
                "d2h_bytes_per_step": int(nfree * 8), "ms_per_step": ms_e2e},
        "roofline": {"bound": "hbm", "kernel": f"k_pcg32 (the solve's FP32 CG iterations: product, two dots and the three "
                               f"updates; {layout}), per iteration of the timed steps, FP64 residuals included",
                     "achieved": bit / (ms_it * 1e-3) / 1e9, "peak": hbm, "unit": "GB/s",
                     "frac": bit / (ms_it * 1e-3) / 1e9 / hbm, "peak_source": "of measured" if pk else "of fallback",
                     "traffic": DRAM_PER_FORMAT_BYTE_PCG32 * fmt_it,
                     "traffic_source": "ncu dram__bytes_read+write of a k_pcg32 launch at 64^3 Q2 per byte of values and "
                                       "vectors, scaled by those bytes",
                     "bytes_per_iteration": bit, "ms_per_iteration": ms_it,
                     "bytes_def": "4*nnz + 36*n (values once; p read, q written; x, r, p, q read, x, r, p written)",
                     "format_bytes_per_iteration": fmt_it, "format_frac": fmt_it / (ms_it * 1e-3) / 1e9 / hbm},
        "roofline_spmv": {"kernel": f"{kname}<float,0> (FP32 SpMV alone, {layout}; not launched by the steps)",
                          "achieved": ach32, "frac": ach32 / hbm, "bytes_per_launch": b32, "ms_per_launch": ms32,
                          "bytes_def": "4*nnz + 8*n (values once, x once, y once)",
                          "format_bytes_per_launch": fmt32, "format_frac": fmt32 / (ms32 * 1e-3) / 1e9 / hbm,
                          "csr_bytes_per_launch": csr_bytes(nfree, nnz, True),
                          "csr_equivalent_gbs": csr_bytes(nfree, nnz, True) / (ms32 * 1e-3) / 1e9},
        "roofline_fp64": {"kernel": f"{kname}<double,0>", "bound": "fp64 pipe (1 DFMA per stored entry)",
                          "achieved_gbs": ach64, "frac_hbm": ach64 / hbm, "bytes_per_launch": b64,
                          "ms_per_launch": ms64, "dfma_per_s": nent / (ms64 * 1e-3),
                          "format_bytes_per_launch": fmt64},
        "cpu_baseline": cb, "clocks": clocks, "gpu_launches": launches,
        "plain_method_32_q1": cfg1, "batch": batch,
    }
    print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
