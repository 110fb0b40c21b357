#!/usr/bin/env python3
"""Benchmark of the GB300 path on the pressure-Poisson workload.

Workload (one "step"): the SIMPLE pressure solve of freeCappuccino on a
128^3 hex mesh of the unit cube (2,097,152 cells) whose interior vertices are
perturbed by U(-0.15h, 0.15h) (seed 42): the implicit Laplacian of
laplacian.f90 with Gamma = 1, Dirichlet on the x=0 patch and Neumann
elsewhere, a N(0,1) right-hand side with its mean removed (seed 43), solved
by the reference's ICCG (DIC-preconditioned CG, linear_solvers.f90:364) from
a zero start to the reference's relative L1 criterion 1e-10.

value  : p-solves/s with matrix, RHS and solution resident in HBM (the whole
         solve, incl. the DIC setup, is one persistent kernel).
e2e    : the same through the C ABI call fc_csrsolve (the csrsolve drop-in)
         with HOST buffers: a, rhs and fi copied in and fi copied out per step.
mixed  : the FP32-inner / FP64-refinement solve to the same FP64 criterion.

`--impl reference` times the reference algorithm on the host cores (the C++
restatement of linear_solvers.f90, single thread like the serial reference).
"""
import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(ROOT, "freecappuccino-dev_gb300")
METRIC = "SIMPLE iters/s & p-solve time to 1e-8 resid, mixed vs FP64 GPU; HBM GB/s"
PERTURB, MESH_SEED, RHS_SEED = 0.15, 42, 43
TOL_REL, ITR_MAX = 1e-10, 20000
L2_BYTES = 129 * 1024 * 1024  # GB300 L2
# relative tolerance of each FP32 inner solve of the mixed-precision runs.
# Multicolour inner ICCG (FC_PREC_MIXED_COLOURED): 1e-5, three refinement steps
# to 1e-10 at 128^3 (the last one only to the reduction still missing).
# Natural-order inner ICCG (FC_PREC_MIXED): 1e-6, two refinement steps.
MIXED_INNER_TOL = 1e-5
MIXED_NATURAL_INNER_TOL = 1e-6


def load_fc():
    import importlib.util
    spec = importlib.util.spec_from_file_location("fcgpu", os.path.join(PKG, "fcgpu.py"))
    mod = importlib.util.module_from_spec(spec)
    sys.modules["fcgpu"] = mod
    spec.loader.exec_module(mod)
    return mod


def rhs(n):
    b = np.random.default_rng(RHS_SEED).standard_normal(n)
    return b - b.mean()


def iccg_bytes_per_iteration(n, nnz):
    """Algorithmic HBM bytes of one FP64 ICCG iteration, each array counted
    once per pass (int32 indices, perfect reuse of gathered vectors):
      SpMV z = A p          12*nnz + 4*(n+1) + 8n (p) + 8n (z)
      DIC forward+backward  12*(nnz-n) + 2*4*(n+1) + 4n (diag) + 8n*4 (r, d, z write, z read)
                            + 8n*3 (backward: d, z read, z write)
      p = z + beta p        8n*3
      x += a p, r -= a z    8n*6
    """
    spmv = 12 * nnz + 4 * (n + 1) + 16 * n
    sweeps = 12 * (nnz - n) + 8 * (n + 1) + 4 * n + 32 * n + 24 * n
    vec = 24 * n + 48 * n
    return spmv + sweeps + vec


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.samples = []
        self.stop = threading.Event()
        self.t = threading.Thread(target=self.run, daemon=True)

    def run(self):
        while not self.stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.Q,
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True,
                                     timeout=5).stdout.strip()
                if out:
                    self.samples.append([v.strip() for v in out.split(",")])
            except Exception:
                pass
            self.stop.wait(0.2)

    def __enter__(self):
        self.t.start()
        return self

    def __exit__(self, *a):
        self.stop.set()
        self.t.join(timeout=10)

    def summary(self):
        if not self.samples:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm = [float(s[1]) for s in self.samples if s[1].replace(".", "").isdigit()]
        mx = [float(s[2]) for s in self.samples if s[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for s in self.samples for k in range(4) if len(s) > 5 + k and
                          s[5 + k].strip().lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.samples)}


def measured_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def profiled_traffic():
    """DRAM bytes per ICCG launch from the committed ncu summary, if any."""
    p = os.path.join(ROOT, "profiles", "iccg_fp64_poisson.md")
    if not os.path.exists(p):
        return None
    for line in open(p):
        if line.startswith("traffic_bytes_per_launch_128:"):
            try:
                return float(line.split(":")[1])
            except ValueError:
                return None
    return None


def cpu_baseline(ia, ja, a, diag, b):
    """The oracle's ICCG (fast build, one core) on the same matrix: one
    whole solve from a zero start to TOL_REL, timed."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_lib
    n = len(diag)
    t0 = time.perf_counter()
    x, r0, info, st = oracle_lib.solve("iccg", ia, ja, a, diag, np.zeros(n), b, ITR_MAX, 0.0, TOL_REL, fast=True)
    dt = time.perf_counter() - t0
    return {"value": 1.0 / dt, "unit": "p-solves/s", "cores": 1, "kind": "port",
            "sample": f"one whole ICCG solve of the same system to 1e-10 ({int(info[0])} iterations, DIC setup and "
                      f"residual included) in {dt:.1f} s (C++ restatement of linear_solvers.f90, -O3, one thread)"}


def progress(msg):
    """A progress line on stderr (the JSON line stays the only stdout)."""
    print(f"[bench {time.strftime('%H:%M:%S')}] {msg}", file=sys.stderr, flush=True)


BATCH_TOL, BATCH_INNER_TOL, BATCH_INNER_ITMAX = 1e-6, 1e-4, 100  # C3b: BiCGStab to 1e-6; FP32 inner settings


def batch_block(fc, args, dev):
    """C3b: independent steady convection-diffusion problems solved together.
    count problems (64, the configuration's count, by default): n^3
    perturbed hex meshes of [0, 2 pi]^3 with
    n ~ U{20..80} (seed 44), cell Peclet number U h / gamma ~ lognormal(0, 1)
    (seed 45), the C4 velocity field and source (tests/cd_cases.py); BiCGStab
    (DILU) to batch_tol relative L1 per problem.  Legs, all on device-resident
    inputs: one batched launch in FP64 (planner's model plan); the mixed
    batched solve (FP32 inner BiCGStab, FP64 refinement) on the model plan
    and on the autotuned plan; the same problems solved one after another (a
    batch of one each) in FP64 and mixed; the tuned mixed batch end to end
    from host buffers.  The CPU estimate is the oracle's BiCGStab (one core)
    timed on the smallest problems and scaled by rows x iterations."""
    import torch
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_lib
    from cd_cases import cd_batch_sizes, cd_batch_system
    ns, pe = cd_batch_sizes(args.batch_count)
    gen = fc.Context(dev)
    probs = [cd_batch_system(fc, gen, int(n), float(p), MESH_SEED + k) for k, (n, p) in enumerate(zip(ns, pe))]
    gen.close()
    np_ = len(probs)
    progress(f"batch: {np_} problems generated")
    rows = np.array([len(p[2]) for p in probs])
    td = torch.device("cuda", dev)
    da = [torch.from_numpy(p[3]).to(td) for p in probs]
    db = [torch.from_numpy(p[4]).to(td) for p in probs]
    xbuf = torch.zeros(int(rows.sum()), dtype=torch.float64, device=td)
    offs = np.concatenate([[0], np.cumsum(rows)])
    dx = [xbuf[offs[k]:offs[k + 1]] for k in range(np_)]
    torch.cuda.synchronize()
    ctx = fc.Context(dev)
    tol, itmax, reps = args.batch_tol, 4000, max(1, args.batch_reps)

    def make(idx):
        B = fc.Batch(ctx)
        for k in idx:
            ia, ja, dg, a, b, xyz = probs[k]
            B.add(ia, ja, dg, xyz)
        B.plan()
        return B

    def run(B, idx):
        xbuf.zero_()
        torch.cuda.synchronize()
        _, infos, st = B.solve([da[k] for k in idx], [dx[k] for k in idx], [db[k] for k in idx], itmax, 0.0, tol,
                               raise_on_error=False)
        if st < 0:
            raise RuntimeError(f"batched solve status {st}: {ctx.error()}")
        return infos

    def timed(groups):
        infos = [None] * np_
        for B, idx in groups:  # warm-up
            run(B, idx)
        ctx.sync()
        ctx.event(0)
        for _ in range(reps):
            xbuf.zero_()
            torch.cuda.synchronize()
            for B, idx in groups:
                _, inf, st = B.solve([da[k] for k in idx], [dx[k] for k in idx], [db[k] for k in idx], itmax, 0.0,
                                     tol, raise_on_error=False)
                if st < 0:
                    raise RuntimeError(f"batched solve status {st}: {ctx.error()}")
                for k, i in zip(idx, inf):
                    infos[k] = i
        ctx.event(1)
        return ctx.elapsed_ms() / reps, infos

    allidx = list(range(np_))
    out = {"problems": np_, "cells": int(rows.sum()), "cells_per_side": [int(v) for v in ns],
           "tol_rel": tol, "solver": "BiCGStab (DILU)"}
    ctx.set_precision(fc.FC_PREC_FP64)
    B = make(allidx)
    out["tiles_model"] = [int(v) for v in B.tiles()]
    out["fp64_batched_ms"], inf64 = timed([(B, allidx)])
    progress(f"batch: fp64 batched {out['fp64_batched_ms']:.1f} ms")
    x64 = [dx[k].cpu().numpy() for k in allidx]
    singles = [(make([k]), [k]) for k in allidx]
    out["fp64_sequential_ms"], _ = timed(singles)
    progress(f"batch: fp64 sequential {out['fp64_sequential_ms']:.1f} ms")
    it64 = np.array([i.itr_used for i in inf64])
    out["fp64_iterations"] = {"min": int(it64.min()), "median": float(np.median(it64)), "max": int(it64.max()),
                              "not_converged": int(sum(i.status != 0 for i in inf64))}
    # FP32 BiCGStab as the reference writes it stalls above 1e-4 on the larger
    # problems: without a cap an inner solve runs to the outer iteration limit
    ctx.set_precision(fc.FC_PREC_MIXED, args.batch_inner_tol, args.batch_inner_itmax)
    out["inner_tol"] = args.batch_inner_tol
    out["inner_itmax"] = args.batch_inner_itmax
    out["mixed_batched_model_ms"], _ = timed([(B, allidx)])
    progress(f"batch: mixed batched (model plan) {out['mixed_batched_model_ms']:.1f} ms")
    a_h = [p[3] for p in probs]
    b_h = [p[4] for p in probs]
    x0 = [np.zeros(len(p[2])) for p in probs]
    tiles, tune_ms = B.tune(a_h, x0, b_h, itmax, 0.0, tol, rounds=args.batch_tune_rounds)
    out["tiles_tuned"] = [int(v) for v in tiles]
    launches0 = ctx.kernel_launches()
    out["mixed_batched_tuned_ms"], infm = timed([(B, allidx)])
    progress(f"batch: mixed batched (tuned plan) {out['mixed_batched_tuned_ms']:.1f} ms")
    out["gpu_launches_per_batched_mixed_solve"] = (ctx.kernel_launches() - launches0) / (reps + 1)
    xm = [dx[k].cpu().numpy() for k in allidx]
    out["mixed_max_rel_diff_vs_fp64"] = float(max(np.abs(u - v).max() / np.abs(v).max() for u, v in zip(xm, x64)))
    # per problem: FP64 iterations, mixed inner iterations and refinement steps
    out["iterations_per_problem"] = {"fp64": [int(i.itr_used) for i in inf64],
                                     "mixed_inner": [int(i.itr_used) for i in infm],
                                     "mixed_outer": [int(i.outer_iterations) for i in infm],
                                     "mixed_group_ms": [float(i.ms) for i in infm]}
    out["mixed_outer_steps_max"] = int(max(i.outer_iterations for i in infm))
    out["mixed_not_converged"] = int(sum(i.status != 0 for i in infm))
    out["mixed_sequential_ms"], _ = timed(singles)
    progress(f"batch: mixed sequential {out['mixed_sequential_ms']:.1f} ms")
    # end to end: host buffers in, solutions back
    ctx.sync()
    ctx.event(0)
    B.solve(a_h, x0, b_h, itmax, 0.0, tol)
    ctx.event(1)
    out["mixed_batched_e2e_ms"] = ctx.elapsed_ms()
    out["e2e_h2d_bytes"] = int(sum(p[3].nbytes + 2 * p[4].nbytes for p in probs))
    out["e2e_d2h_bytes"] = int(sum(p[4].nbytes for p in probs))
    out["speedup_mixed_batched_vs_fp64_sequential"] = out["fp64_sequential_ms"] / out["mixed_batched_tuned_ms"]
    for b_, _ in singles:
        b_.close()
    B.close()
    ctx.set_precision(fc.FC_PREC_FP64)
    ctx.close()
    if not args.no_cpu:
        order = np.argsort(rows)
        done_rows_iters, t_cpu, used = 0.0, 0.0, []
        for k in order:
            ia, ja, dg, a, b, _ = probs[k]
            t0 = time.perf_counter()
            x, r0, info, st = oracle_lib.solve("bicgstab", ia, ja, a, dg, np.zeros(len(dg)), b, itmax, 0.0, tol,
                                               fast=True)
            t_cpu += time.perf_counter() - t0
            done_rows_iters += len(dg) * max(1, int(info[0]))
            used.append(int(ns[k]))
            if t_cpu > args.batch_cpu_seconds:
                break
        per = t_cpu / done_rows_iters
        est = per * float((rows * it64).sum()) * 1e3
        out["cpu_sequential_ms_est"] = est
        out["cpu_sample"] = (f"oracle BiCGStab (C++ restatement, -O3, one thread) on the {len(used)} smallest "
                             f"problems (n = {used[0]}..{used[-1]}) in {t_cpu:.1f} s, scaled by rows x the FP64 "
                             f"GPU iteration counts of all {np_} problems")
        out["speedup_mixed_batched_vs_cpu"] = est / out["mixed_batched_tuned_ms"]
    return out


def workload_config(n, cells, nnz):
    """The `config` of both arms: the workload and how the timed region
    relates to L2 (inputs larger than L2, or not)."""
    work_bytes = 12 * nnz + 4 * (cells + 1) + 8 * 8 * cells
    l2_note = (f"inputs larger than L2 (matrix + vectors ~{work_bytes / 1e9:.2f} GB)" if work_bytes > L2_BYTES
               else f"inputs of ~{work_bytes / 1e6:.0f} MB fit in L2: not a contract-size measurement")
    return {"workload": f"{n}^3 perturbed-hex pressure Poisson, ICCG (DIC) FP64 to 1e-10 rel. L1",
            "cells": int(cells), "nnz": int(nnz), "l2": l2_note}


def run_reference(args, rank, world):
    """The reference's ICCG (the oracle: C++ restatement of
    linear_solvers.f90:364-545, -O3, one thread like the serial reference) on
    the same system, built without the GPU library (numpy box generator +
    the oracle's geometry, CSR and Laplacian).  Each timed step is one whole
    solve from a zero start to the 1e-10 relative L1 criterion, its
    iterations counted by the solver; each warm-up step is the DIC setup and
    a few iterations of the same system."""
    if rank != 0:
        return
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_lib
    from box_mesh import hex_box
    n = args.n
    arrays = hex_box(n, n, n, perturb=PERTURB, seed=MESH_SEED)
    oc = oracle_lib.Case(arrays, fast=True)
    b = rhs(oc.numCells)
    oc.set("su", b)
    oc.laplacian(np.ones(oc.numCells), np.zeros(oc.numTotal), 0b1)
    ia, ja, a, dg = oc.get_int("ia"), oc.get_int("ja"), oc.get("a"), oc.get_int("diag")
    nc = oc.numCells
    for _ in range(args.warmup):
        oracle_lib.solve("iccg", ia, ja, a, dg, np.zeros(nc), b, args.ref_warmup_iters, 0.0, 1e-30, fast=True)
    per, iters = [], []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        x, r0, info, st = oracle_lib.solve("iccg", ia, ja, a, dg, np.zeros(nc), b, ITR_MAX, 0.0, TOL_REL, fast=True)
        per.append(time.perf_counter() - t0)
        iters.append(int(info[0]))
        if st != 0 or not (info[2] / (info[1] + 1e-20) < TOL_REL):
            raise RuntimeError(f"reference ICCG did not converge: status {st}, info {info}")
    total = float(np.sum(per))
    value = args.steps / total
    sample = (f"each step one whole ICCG solve of the {n}^3 system to 1e-10 relative L1 from a zero start "
              f"({iters[0]} iterations, C++ restatement of linear_solvers.f90, -O3, one thread); warm-up steps: "
              f"DIC setup + {args.ref_warmup_iters} iterations")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "p-solves/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": total / args.steps * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": workload_config(n, nc, len(ja)),
            "iterations_per_solve": iters,
            "cpu_baseline": {"value": value, "unit": "p-solves/s", "cores": 1, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": "p-solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


LID_PATCH = 3  # ymax patch of the box generator (xmin, xmax, ymin, ymax, zmin, zmax)


def cavity_fields(m, nT, nC):
    """Initial fields of the lid-driven cavity: lid u = 1 on the y = 1 wall."""
    a = m.arrays()
    u = np.zeros(nT)
    st = a["startFace"][LID_PATCH] - m.numInnerFaces
    u[nC + st:nC + st + a["nfaces"][LID_PATCH]] = 1.0
    nwal = int(sum(nf for t, nf in zip(a["bctype"], a["nfaces"]) if t == 1))
    return a, u, nwal


def simple_iterations(n=128, iters=4, perturb=PERTURB, dev=0, tets=False, viscos=0.01, scheme=1, grad=0,
                      urf=(0.8, 0.3)):
    """`iters` FP64 SIMPLE iterations of the n^3 lid-driven cavity of the
    SIMPLE leg (perturbed hexes, seed MESH_SEED; `tets` splits every hex into
    6 tetrahedra): the command the kernel launch lists and ncu captures of
    one SIMPLE iteration run, e.g.
    python -c "import bench; bench.simple_iterations(128, 4)", or for the
    6M-tet cavity of the C5 leg (Re 400, boundedLinearUpwind, LSQ gradients)
    python -c "import bench; bench.simple_iterations(100, 3, tets=True, viscos=1/400, scheme=19, grad=1, urf=(0.6, 0.2))".
    Returns the last iteration's resor."""
    fc = load_fc()
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=perturb, seed=MESH_SEED, tets=tets)
    nC, nT = m.numCells, m.numTotal
    _, u, nwal = cavity_fields(m, nT, nC)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    zero = np.zeros(nT)
    for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, viscos)).items():
        ctx.field_set(k, v)
    ctx.field_set("visw", np.full(max(nwal, 1), viscos))
    for k in ("flmass", "a", "dUdxi", "dVdxi", "dWdxi", "dPdxi"):
        ctx.field_fill(k, 0.0)
    ctx.simple_params(fc.SimpleParams.cavity(viscos=viscos, scheme=scheme, grad=grad, urfU=urf[0], urfP=urf[1]))
    ctx.init_flmass()
    r = None
    for _ in range(iters):
        r = ctx.simple_iteration()
    ctx.sync()
    print("simple_iterations", n, iters, "launches", ctx.kernel_launches(), "resor", list(r), flush=True)
    ctx.close()
    return r


TURB_VISCOS = 1e-3  # Re 1000 cavity for the turbulence leg


def turbulent_cavity(fc, n, dev=0):
    """The n^3 perturbed lid-driven cavity at Re 1000 with the k-omega SST
    model (TurbModelData.f90 defaults; k = 1e-4 and omega = 1 everywhere at
    the start), its wall distance computed: (fc.Mesh, context, arrays)."""
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=PERTURB, seed=MESH_SEED)
    nC, nT = m.numCells, m.numTotal
    a, u, nwal = cavity_fields(m, nT, nC)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    zero = np.zeros(nT)
    for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, TURB_VISCOS),
                     te=np.full(nT, 1e-4), ed=np.full(nT, 1.0)).items():
        ctx.field_set(k, v)
    ctx.field_set("visw", np.full(max(nwal, 1), TURB_VISCOS))
    for k in ("flmass", "a", "dUdxi", "dVdxi", "dWdxi", "dPdxi", "fsst"):
        ctx.field_fill(k, 0.0)
    ctx.simple_params(fc.SimpleParams.cavity(viscos=TURB_VISCOS))
    ctx.turbulence_params(fc.TurbulenceParams.defaults())
    ctx.init_flmass()
    ctx.wall_distance()
    return m, ctx, a


def turbulence_iterations(n=128, iters=3, dev=0):
    """`iters` SIMPLE iterations each followed by the k-omega SST update on
    the turbulent cavity: the command the launch lists and ncu captures of
    the turbulence kernels run, e.g.
    python -c "import bench; bench.turbulence_iterations(128, 3)"."""
    fc = load_fc()
    m, ctx, _ = turbulent_cavity(fc, n, dev)
    for _ in range(iters):
        ctx.simple_iteration()
        r = ctx.kw_sst()
    ctx.sync()
    print("turbulence_iterations", n, iters, "resor56", list(r), flush=True)
    ctx.close()


def batch_solves(count=64, mixed=False, dev=0):
    """One batched BiCGStab(DILU) solve of the first `count` problems of the
    C3b set (FP64, or with `mixed` the FP32-inner / FP64-refinement solve with
    the bench's inner settings) after one untimed solve: the command of the
    batched kernels' launch list and ncu captures, e.g.
    python -c "import bench; bench.batch_solves(8)"."""
    import torch
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from cd_cases import cd_batch_sizes, cd_batch_system
    fc = load_fc()
    ns, pe = cd_batch_sizes(count)
    gen = fc.Context(dev)
    probs = [cd_batch_system(fc, gen, int(n), float(q), MESH_SEED + k) for k, (n, q) in enumerate(zip(ns, pe))]
    gen.close()
    td = torch.device("cuda", dev)
    da = [torch.from_numpy(p[3]).to(td) for p in probs]
    db = [torch.from_numpy(p[4]).to(td) for p in probs]
    dx = [torch.zeros(len(p[2]), dtype=torch.float64, device=td) for p in probs]
    ctx = fc.Context(dev)
    if mixed:
        ctx.set_precision(fc.FC_PREC_MIXED, BATCH_INNER_TOL, BATCH_INNER_ITMAX)
    B = fc.Batch(ctx)
    for ia, ja, dg, a, b, xyz in probs:
        B.add(ia, ja, dg, xyz)
    B.plan()
    for _ in range(2):
        for x in dx:
            x.zero_()
        _, infos, st = B.solve(da, dx, db, 4000, 0.0, BATCH_TOL, raise_on_error=False)
    ctx.sync()
    print("batch_solves", count, "mixed" if mixed else "fp64", "status", st,
          "iterations", [int(i.itr_used) for i in infos], flush=True)
    B.close()
    ctx.close()


def adjoint_solves(n=96, calls=2, dev=0):
    """`calls` passes of the C4 adjoint on the n^3 mesh: assembly
    (fc_cd_assemble), the forward BiCGStab(DILU) solve, the objective and the
    adjoint (transposed solve and reverse face loop): the command of the
    adjoint kernels' launch list and ncu captures, e.g.
    python -c "import bench; bench.adjoint_solves(96, 2)"."""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from cd_cases import TWO_PI, cd_inputs, cd_objective, cd_source
    fc = load_fc()
    m = fc.Mesh.box(n, n, n, TWO_PI, TWO_PI, TWO_PI, perturb=PERTURB, seed=MESH_SEED)
    _, fm, gamma = cd_inputs(fc, m)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    ctx.field_set("flmass", fm)
    xc, yc, zc = ctx.geometry("xc"), ctx.geometry("yc"), ctx.geometry("zc")
    vol = ctx.geometry("vol")
    src = cd_source(xc, yc, zc)
    for _ in range(calls):
        ctx.cd_assemble(gamma, src)
        phi, finfo = ctx.cd_solve(2000, 1e-6)
        J, g = cd_objective(phi, vol, xc)
        lam, grad, ainfo = ctx.cd_adjoint(g, 2000, 1e-6)
    ctx.sync()
    print("adjoint_solves", n, calls, "J", J, "iterations", finfo.itr_used, ainfo.itr_used, flush=True)
    ctx.close()


def mesh_setup(n=100, tets=True, perturb=PERTURB, dev=0):
    """fc_set_mesh of the n^3 perturbed box (6 tetrahedra per hex when
    `tets`): wall-clock seconds of the host mesh generation, of set_mesh and
    of its phases (fc_get_setup_times), e.g.
    python -c "import bench; bench.mesh_setup(100, True)" (6,000,000 cells)."""
    fc = load_fc()
    t0 = time.perf_counter()
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=perturb, seed=MESH_SEED, tets=tets)
    t_box = time.perf_counter() - t0
    ctx = fc.Context(dev)
    t0 = time.perf_counter()
    ctx.set_mesh(m)
    ctx.sync()
    out = {"cells": m.numCells, "mesh_box_host": round(t_box, 3), "fc_set_mesh": round(time.perf_counter() - t0, 3),
           "phases": {k: round(v, 3) for k, v in ctx.setup_times().items()}}
    ctx.close()
    print(json.dumps(out), flush=True)
    return out


def temperature_iterations(n=128, iters=3, dev=0):
    """`iters` SIMPLE iterations each followed by calculate_temperature on the
    n^3 perturbed cavity with the hot lid (isothermal lid at T = 1, the other
    walls adiabatic, temperature.f90's defaults): the command the profiles of
    the temperature kernels run, e.g.
    python -c "import bench; bench.temperature_iterations(128, 3)"."""
    fc = load_fc()
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=PERTURB, seed=MESH_SEED)
    nC, nT = m.numCells, m.numTotal
    a, u, nwal = cavity_fields(m, nT, nC)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    zero = np.zeros(nT)
    t = np.zeros(nT)
    st = a["startFace"][LID_PATCH] - m.numInnerFaces
    t[nC + st:nC + st + a["nfaces"][LID_PATCH]] = 1.0
    for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, 0.01), t=t).items():
        ctx.field_set(k, v)
    ctx.field_set("visw", np.full(max(nwal, 1), 0.01))
    for k in ("flmass", "a", "dUdxi", "dVdxi", "dWdxi", "dPdxi", "dTdxi"):
        ctx.field_fill(k, 0.0)
    ctx.simple_params(fc.SimpleParams.cavity(viscos=0.01))
    bcdf = np.zeros(len(a["bctype"]))
    bcdf[LID_PATCH] = 1.0
    ctx.temperature_params(fc.TemperatureParams.defaults(), bcdf)
    ctx.init_flmass()
    for _ in range(iters):
        ctx.simple_iteration()
        r7 = ctx.calculate_temperature()
    ctx.sync()
    print("temperature_iterations", n, iters, "resor7", r7, flush=True)
    ctx.close()


def turbulence_block(fc, args, dev, with_cpu):
    """f2: the k-omega SST update (fc_kw_sst: strain, k and omega equations
    with BiCGStab, eddy viscosity) on the n^3 turbulent cavity after a few
    SIMPLE + SST iterations; event time per call, and the oracle's update of
    the same state on one core."""
    n = args.turb_n
    m, ctx, a = turbulent_cavity(fc, n, dev)
    for _ in range(3):
        ctx.simple_iteration()
        ctx.kw_sst()
    state = {k: ctx.field_get(k) for k in ("u", "v", "w", "p", "flmass", "vis", "te", "ed", "fsst", "visw",
                                            "walldist")}
    ctx.sync()
    ctx.event(0)
    for _ in range(args.turb_calls):
        r = ctx.kw_sst()
    ctx.event(1)
    ms = ctx.elapsed_ms() / args.turb_calls
    out = {"workload": f"{n}^3 perturbed lid-driven cavity, Re {1.0 / TURB_VISCOS:g}, k-omega SST (high-Re, wall "
                       "functions), BiCGStab(DILU) for k and omega (maxiter 10, tolRel 0.01)",
           "cells": m.numCells, "kw_sst_ms": ms, "kw_sst_per_s": 1e3 / ms, "resor56": [float(v) for v in r],
           "calls": args.turb_calls}
    ctx.close()
    if with_cpu:
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import oracle_lib
        oc = oracle_lib.Case(a, fast=True)
        for k, v in state.items():
            oc.set(k, v)
        oc.set("den", np.ones(m.numTotal))
        oc.param("viscos", TURB_VISCOS)
        t0 = time.perf_counter()
        oc.kw_sst()
        dt = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": 1.0 / dt, "unit": "SST updates/s", "cores": 1, "kind": "port",
                               "sample": "one k-omega SST update of the same state (C++ restatement, -O3, one thread)"}
        out["gpu_vs_cpu"] = out["kw_sst_per_s"] / out["cpu_baseline"]["value"]
    return out


def simple_block(fc, args, dev, with_cpu, n, perturb=0.0, cpu_skip=None, tets=False, viscos=0.01, scheme=1, grad=0,
                 iters=None, cpu_iters=None, urf=(0.8, 0.3), momentum_batch=False, skip=None):
    """SIMPLE iterations per second on the n^3 lid-driven cavity (unit cube,
    nu = 0.01, central differencing with deferred correction, Gauss gradients,
    BiCGStab(DILU) for U, ICCG(DIC) for p, the settings of
    examples/cavity/input.nml), FP64 and mixed precision, plus the oracle's
    SIMPLE iteration on one core.  perturb > 0 moves the interior vertices by
    U(-perturb h, perturb h) (seed 42): the non-orthogonal mesh."""
    t0 = time.perf_counter()
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=perturb, seed=MESH_SEED, tets=tets)
    t_box = time.perf_counter() - t0
    iters = args.simple_iters if iters is None else iters
    skip = args.simple_skip if skip is None else skip
    cpu_iters = args.simple_cpu_iters if cpu_iters is None else cpu_iters
    nC, nT = m.numCells, m.numTotal
    a, u, nwal = cavity_fields(m, nT, nC)
    ctx = fc.Context(dev)
    t0 = time.perf_counter()
    ctx.set_mesh(m)
    ctx.sync()
    t_set = time.perf_counter() - t0
    prm = fc.SimpleParams.cavity(viscos=viscos, scheme=scheme, grad=grad, urfU=urf[0], urfP=urf[1])

    def reset():
        zero = np.zeros(nT)
        for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, viscos)).items():
            ctx.field_set(k, v)
        ctx.field_set("visw", np.full(max(nwal, 1), viscos))
        for k in ("flmass", "a", "dUdxi", "dVdxi", "dWdxi", "dPdxi"):
            ctx.field_fill(k, 0.0)
        ctx.simple_params(prm)
        ctx.init_flmass()

    mesh_kind = f"perturbed hexes (+-{perturb:g} h)" if perturb > 0 else "uniform hexes"
    if tets:
        mesh_kind += " split into 6 tetrahedra each"
    sname = {1: "central", 19: "boundedLinearUpwind"}.get(scheme, str(scheme))
    gname = {0: "Gauss", 1: "LSQ", 2: "LSQ_DM"}[grad]
    out = {"workload": f"{n}^3 lid-driven cavity on {mesh_kind}, Re={1.0 / viscos:g}, SIMPLE ({sname}/DC, {gname}, "
                       f"BiCGStab U, ICCG p, urfU {urf[0]:g}, urfP {urf[1]:g})", "cells": nC, "unit": "SIMPLE iters/s",
           "setup_s": {"mesh_box_host": round(t_box, 2), "fc_set_mesh": round(t_set, 2),
                       "fc_set_mesh_phases": {k: round(v, 3) for k, v in ctx.setup_times().items()}}}
    for mode, key in ((fc.FC_PREC_FP64, "value"), (fc.FC_PREC_MIXED_COLOURED, "mixed")):
        ctx.set_precision(mode, MIXED_INNER_TOL, 0) if mode else ctx.set_precision(mode)
        reset()
        for _ in range(skip):
            ctx.simple_iteration()
        ctx.sync()
        ctx.event(0)
        done, err = 0, None
        for _ in range(iters):
            try:
                res = ctx.simple_iteration()
            except fc.FcError as e:  # a diverging run ends the timed loop
                err = str(e)
                break
            done += 1
        ctx.event(1)
        ms = ctx.elapsed_ms() / max(done, 1)
        out[key] = 1e3 / ms
        out[key + "_ms_per_iteration"] = ms
        out[key + "_resor"] = [float(v) for v in res] if done else None
        if err:
            out[key + "_stopped"] = f"after {done} of {iters} iterations: {err}"
            progress(f"simple {n}^3 {key}: stopped after {done} iterations: {err}")
    if momentum_batch:
        # C3a: the three momentum solves of calcuvw (shared off-diagonals, three
        # diagonals and sources) one after another and as one batched launch,
        # on the field developed by the untimed iterations; calcuvw = assembly +
        # the three solves, timed alone, then whole SIMPLE iterations
        ctx.set_precision(fc.FC_PREC_FP64)
        reset()
        for _ in range(max(skip, 10)):
            ctx.simple_iteration()
        c3 = {"workload": "calcuvw on the developed field: momentum assembly + U, V, W BiCGStab(DILU) solves, "
                          f"maxiterU {prm.maxiterU}, tolRelU {prm.tolRelU:g}"}
        for on, key in ((False, "sequential"), (True, "batched")):
            ctx.simple_batched_momentum(on)
            ctx.calcuvw()  # warm-up (builds the three systems on the first batched call)
            ctx.sync()
            ctx.event(0)
            for _ in range(args.momentum_calls):
                ctx.calcuvw()
            ctx.event(1)
            c3[key + "_calcuvw_ms"] = ctx.elapsed_ms() / args.momentum_calls
            progress(f"momentum: {key} calcuvw {c3[key + '_calcuvw_ms']:.2f} ms")
        ctx.event(0)
        for _ in range(iters):
            res = ctx.simple_iteration()
        ctx.event(1)
        ms = ctx.elapsed_ms() / iters
        ctx.simple_batched_momentum(False)
        c3["speedup_calcuvw"] = c3["sequential_calcuvw_ms"] / c3["batched_calcuvw_ms"]
        out["momentum_batched"] = c3
        out["value_batched_momentum"] = 1e3 / ms
        out["value_batched_momentum_ms_per_iteration"] = ms
        out["value_batched_momentum_resor"] = [float(v) for v in res]
    out["iterations_timed"] = f"{iters} after {skip} untimed"
    out["mixed_note"] = ("ICCG for p with the multicolour FP32 inner solve, capped at maxiterP iterations as the "
                         "reference caps it: it reduces the p residual less per SIMPLE iteration than the "
                         "natural-order DIC, so the *_resor after the same iterations differ")
    ctx.set_precision(fc.FC_PREC_FP64)
    ctx.close()
    if with_cpu:
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import oracle_lib
        oc = oracle_lib.Case(a, fast=True)
        zero = np.zeros(nT)
        for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, viscos)).items():
            oc.set(k, v)
        if nwal:
            oc.set("visw", np.full(nwal, viscos))
        for k in ("flmass", "a"):
            oc.set(k, np.zeros(oc._len(k)))
        for k in ("dUdxi", "dVdxi", "dWdxi", "dPdxi"):
            oc.set(k, np.zeros(3 * nT))
        for name in ("viscos", "densit", "urfP", "gdsU", "cSchemeU", "pscheme", "maxiterU", "maxiterP", "npcor",
                     "pRefCell", "tolAbsU", "tolRelU", "tolAbsP", "tolRelP", "gradScheme"):
            oc.param(name, getattr(prm, name))
        for i in range(3):
            oc.param(f"urfU{i + 1}", prm.urfU[i])
        oc.solver("U", prm.lSolverU.decode())
        oc.solver("P", prm.lSolverP.decode())
        oc.L.orc_init_flmass(oc.h)
        skip = args.simple_skip if cpu_skip is None else cpu_skip
        for _ in range(skip):
            oc.simple_iteration()
        t0 = time.perf_counter()
        for _ in range(cpu_iters):
            oc.simple_iteration()
        dt = (time.perf_counter() - t0) / cpu_iters
        out["cpu_baseline"] = {"value": 1.0 / dt, "unit": "SIMPLE iters/s", "cores": 1, "kind": "port",
                               "sample": f"{cpu_iters} SIMPLE iterations of the same cavity after "
                                         f"{skip} untimed (C++ restatement, -O3, one thread)"}
        out["gpu_fp64_vs_cpu"] = out["value"] / out["cpu_baseline"]["value"]
    return out


def piso_block(fc, args, dev, with_cpu):
    """PISO time steps (Euler, ncorr 2, one pressure solve per corrector,
    urf 1) of the n^3 perturbed lid-driven cavity from rest, dt = 0.1 h:
    milliseconds per time step (time_shift + calcuvw + calcp_piso) on the
    GPU in FP64 and the oracle's time step on one core (opt-in: --piso-n)."""
    n = args.piso_n
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=PERTURB, seed=MESH_SEED)
    nC, nT = m.numCells, m.numTotal
    a, u, nwal = cavity_fields(m, nT, nC)
    dt = 0.1 / n
    kw = dict(urfU=1.0, urfP=1.0, maxiterU=20, maxiterP=100, tolRelU=1e-6, tolRelP=1e-6)
    prm = fc.SimpleParams.cavity(**kw)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    zero = np.zeros(nT)
    for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, 0.01)).items():
        ctx.field_set(k, v)
    ctx.field_set("visw", np.full(max(nwal, 1), 0.01))
    ctx.simple_params(prm)
    ctx.transient_params(dt, fc.FC_TIME_BDF, 1, 2)
    ctx.init_flmass()
    for _ in range(2):
        ctx.time_shift()
        ctx.piso_iteration()
    ctx.sync()
    ctx.event(0)
    for _ in range(args.piso_steps):
        ctx.time_shift()
        res = ctx.piso_iteration()
    ctx.event(1)
    ms = ctx.elapsed_ms() / args.piso_steps
    ctx.close()
    out = {"workload": f"{n}^3 perturbed lid-driven cavity from rest, PISO (Euler, dt {dt:g}, ncorr 2, npcor 1), "
                       "BiCGStab U / ICCG p to 1e-6", "cells": nC, "ms_per_time_step": ms,
           "resor_last": [float(v) for v in res], "steps_timed": f"{args.piso_steps} after 2 untimed"}
    if with_cpu:
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import oracle_lib
        oc = oracle_lib.Case(a, fast=True)
        for k, v in dict(u=u, v=zero, w=zero, p=zero, pp=zero, den=np.ones(nT), vis=np.full(nT, 0.01)).items():
            oc.set(k, v)
        if nwal:
            oc.set("visw", np.full(nwal, 0.01))
        for name in ("viscos", "densit", "urfP", "gdsU", "cSchemeU", "pscheme", "maxiterU", "maxiterP", "npcor",
                     "pRefCell", "tolAbsU", "tolRelU", "tolAbsP", "tolRelP", "gradScheme"):
            oc.param(name, getattr(prm, name))
        for i in range(3):
            oc.param(f"urfU{i + 1}", prm.urfU[i])
        for k, v in dict(timestep=dt, tscheme=1, piso=1, ncorr=2).items():
            oc.param(k, v)
        oc.solver("U", prm.lSolverU.decode())
        oc.solver("P", prm.lSolverP.decode())
        oc.L.orc_init_flmass(oc.h)
        oc.time_shift()
        oc.piso_iteration()
        t0 = time.perf_counter()
        oc.time_shift()
        oc.piso_iteration()
        dtc = time.perf_counter() - t0
        out["cpu_baseline"] = {"value": dtc * 1e3, "unit": "ms per time step", "cores": 1, "kind": "port",
                               "sample": "the second time step of the same run (C++ restatement, -O3, one thread)"}
        out["gpu_vs_cpu"] = dtc * 1e3 / ms
    return out


def spmv_leg(fc, ctx, nC, calls):
    """FP64 y = A x through fc_spmv (ax_cr) on device-resident arrays of the
    same 128^3 system: the per-call CUDA-event time includes the call's host
    work and its stream synchronisation, so it bounds the kernel time from
    above; ncu's launch list gives the kernel alone."""
    import torch
    ia, ja, dg, _, _ = ctx.csr_pattern()
    dev = torch.device("cuda", torch.cuda.current_device())
    tia, tja, tdg = (torch.from_numpy(np.ascontiguousarray(v, dtype=np.int32)).to(dev) for v in (ia, ja, dg))
    ta = torch.from_numpy(ctx.field_get("a")).to(dev)
    tx = torch.from_numpy(np.random.default_rng(RHS_SEED).standard_normal(nC)).to(dev)
    ty = torch.zeros(nC, dtype=torch.float64, device=dev)

    def call():
        st = ctx.L.fc_spmv(ctx.h, nC, len(ja), fc._ptr(tia), fc._ptr(tja), fc._ptr(ta), fc._ptr(tdg), fc._ptr(tx),
                           fc._ptr(ty), 0)
        if st != 0:
            raise RuntimeError(f"fc_spmv status {st}")

    for _ in range(3):
        call()
    ms = []
    for _ in range(calls):
        ctx.event(0)
        call()
        ctx.event(1)
        ms.append(ctx.elapsed_ms())
    us = float(np.median(ms)) * 1e3
    nbytes = 12 * len(ja) + 4 * (nC + 1) + 16 * nC
    return {"calls": calls, "us_per_call": us, "algorithmic_bytes": nbytes,
            "gbs_per_call": nbytes / (us * 1e-6) / 1e9,
            "note": "per call, host work and the call's synchronisation included (upper bound on the kernel)"}


def gradient_block(fc, args, dev):
    """Gradient kernels on the n^3 perturbed hex mesh (128^3: 2,097,152
    cells): fc_grad on a device-resident smooth field for Gauss, LSQ,
    LSQ_DM, their exact 3x3 forms and the node-based Gauss gradient, and
    Gauss with each slope limiter.  Event time per call (the limiter and
    node-gradient calls include their extra passes); minimal bytes = the
    field and the geometry each gradient reads once plus the gradient it
    writes, for a bandwidth figure."""
    n = args.grad_n
    m = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=PERTURB, seed=MESH_SEED)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    nC, nI, nF, nT = m.numCells, m.numInnerFaces, m.numFaces, m.numTotal
    xc, yc, zc = ctx.geometry("xc"), ctx.geometry("yc"), ctx.geometry("zc")
    phi = np.zeros(nT)
    phi[:nC] = np.sin(3 * xc) * np.cos(2 * yc) + zc * zc
    ctx.field_set("u", phi)
    pu, pg = ctx.field_ptr("u"), ctx.field_ptr("dUdxi")
    # gauss: phi, owner/neighbour, area vectors, facint, vol in; g out
    gauss_bytes = 8 * nT + 4 * (nF + nI) + 24 * nF + 8 * nI + 8 * nC + 24 * nT
    lsq_bytes = 8 * nT + 4 * (nF + nI) + 24 * nF + 72 * nC + 24 * nT  # face centres or cell centres, D matrix

    def timed(scheme, calls):
        def call():
            st = ctx.L.fc_grad(ctx.h, scheme, pu, pg)
            if st != 0:
                raise RuntimeError(f"fc_grad({scheme}) status {st}: {ctx.error()}")
        for _ in range(3):
            call()
        ctx.sync()
        ctx.event(0)
        for _ in range(calls):
            call()
        ctx.event(1)
        return ctx.elapsed_ms() / calls

    out = {"workload": f"{n}^3 perturbed hexes (+-{PERTURB:g} h), smooth field, fc_grad on device arrays",
           "cells": nC, "calls": args.grad_calls}
    for name, scheme, nbytes in (("gauss", fc.FC_GRAD_GAUSS, gauss_bytes), ("lsq", fc.FC_GRAD_LSQ, lsq_bytes),
                                 ("lsq_dm", fc.FC_GRAD_LSQ_DM, lsq_bytes),
                                 ("lsq_exact", fc.FC_GRAD_LSQ_EXACT, lsq_bytes),
                                 ("lsq_dm_exact", fc.FC_GRAD_LSQ_DM_EXACT, lsq_bytes),
                                 ("node_gauss", fc.FC_GRAD_NODE_GAUSS, None)):
        ms = timed(scheme, args.grad_calls)
        out[name + "_ms"] = ms
        if nbytes:
            out[name + "_min_bytes_gbs"] = nbytes / (ms * 1e-3) / 1e9
    for name, kind in (("barth_jespersen", fc.FC_LIMITER_BJ), ("venkatakrishnan", fc.FC_LIMITER_VENKAT),
                       ("r3", fc.FC_LIMITER_R), ("multidimensional", fc.FC_LIMITER_MD)):
        ctx.set_gradient_limiter(kind)
        out["gauss_" + name + "_ms"] = timed(fc.FC_GRAD_GAUSS, args.grad_calls)
    ctx.set_gradient_limiter(fc.FC_LIMITER_NONE)
    ctx.close()
    return out


def adjoint_block(fc, args, dev):
    """C4: discrete adjoint of steady convection-diffusion on the n^3
    perturbed hex mesh of [0, 2 pi]^3: u = 0.5 (sin x cos y, -cos x sin y, 0)
    (face fluxes of the stream function), lognormal diffusivity (mu -4,
    sigma 0.5, seed 46), a Gaussian source blob at (pi, pi, pi) with sigma 0.5,
    J = volume-weighted mean of phi^2 over x > pi.  Times the forward solve and
    the adjoint (transposed solve + reverse face loop) and checks dJ/dgamma by
    central differences of J along fd_dirs smooth random directions
    gamma (1 +- h v), v a product of random low-frequency sines (seed 47),
    h = 1e-2, each side a full re-solve.  (Single-cell differences need
    solves far below the residual at which BiCGStab as the reference writes it
    stalls at this size; they are checked on small meshes by the tests.)"""
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    from cd_cases import TWO_PI, cd_inputs, cd_objective, cd_source
    n = args.adjoint_n
    m = fc.Mesh.box(n, n, n, TWO_PI, TWO_PI, TWO_PI, perturb=PERTURB, seed=MESH_SEED)
    a, fm, gamma = cd_inputs(fc, m)
    ctx = fc.Context(dev)
    ctx.set_mesh(m)
    ctx.field_set("flmass", fm)
    xc, yc, zc = ctx.geometry("xc"), ctx.geometry("yc"), ctx.geometry("zc")
    vol = ctx.geometry("vol")
    src = cd_source(xc, yc, zc)
    tol, itmax = 1e-6, 2000

    def J_of(gm):
        ctx.cd_assemble(gm, src)
        phi, info = ctx.cd_solve(itmax, tol)
        if info.status != 0:
            raise RuntimeError(f"convection-diffusion solve status {info.status}")
        return phi, info

    for _ in range(2):  # warm-up
        phi, finfo = J_of(gamma)
        J, g = cd_objective(phi, vol, xc)
        lam, grad, ainfo = ctx.cd_adjoint(g, itmax, tol)
    ctx.sync()
    ctx.event(0)
    ctx.cd_assemble(gamma, src)
    ctx.event(1)
    asm_ms = ctx.elapsed_ms()
    phi, finfo = J_of(gamma)
    J, g = cd_objective(phi, vol, xc)
    ctx.event(0)
    lam, grad, ainfo = ctx.cd_adjoint(g, itmax, tol)
    ctx.event(1)
    adj_ms = ctx.elapsed_ms()
    if ainfo.status != 0:
        raise RuntimeError(f"adjoint solve status {ainfo.status}")
    # the reverse face loop against the oracle's cd_gradient on the same phi
    # and lambda, at this size (one face loop on the host)
    oracle_diff = None
    if not args.no_cpu:
        import oracle_lib
        oc = oracle_lib.Case(a)
        oc.set("flmass", fm)
        go = oc.cd_gradient(phi, lam)
        oracle_diff = float(np.abs(grad - go).max() / max(np.abs(go).max(), 1e-300))
        del oc
    rng = np.random.default_rng(47)
    h, rel = 1e-2, []
    for _ in range(args.adjoint_fd_dirs):
        k = rng.integers(1, 4, 3)
        ph = rng.uniform(0.0, 2.0 * np.pi, 3)
        v = np.sin(k[0] * xc + ph[0]) * np.sin(k[1] * yc + ph[1]) * np.sin(k[2] * zc + ph[2])
        Jp = cd_objective(J_of(gamma * (1.0 + h * v))[0], vol, xc)[0]
        Jm = cd_objective(J_of(gamma * (1.0 - h * v))[0], vol, xc)[0]
        fd = (Jp - Jm) / (2.0 * h)
        ad = float(np.dot(grad, gamma * v))
        rel.append(abs(fd - ad) / max(abs(fd), 1e-300))
    ctx.close()
    return {"workload": f"{n}^3 perturbed hexes on [0,2pi]^3, steady convection-diffusion, lognormal gamma, "
                        f"J = mean phi^2 over x > pi", "cells": m.numCells, "J": J,
            "assemble_ms": asm_ms, "forward_solve_ms": finfo.ms, "forward_iterations": finfo.itr_used,
            "adjoint_ms": adj_ms, "adjoint_solve_ms": ainfo.ms, "adjoint_iterations": ainfo.itr_used,
            "solver": f"BiCGStab(DILU) FP64 to {tol:g} relative L1 (forward and transposed)",
            "fd_directions": len(rel), "fd_step": "gamma (1 +- 1e-2 v), full re-solves",
            "fd_max_rel_err": float(max(rel)), "fd_median_rel_err": float(np.median(rel)),
            "oracle_gradient_max_rel_diff": oracle_diff}


def max_over_ranks(dist, x):
    """x maximised over the ranks of the process group (x itself without one)."""
    if not dist:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t[0])


def replica_throughput(world, steps, elapsed_ms):
    """Whole-job solves per second of independent replicas: every rank solves
    `steps` systems, elapsed_ms is the slowest rank's time."""
    return world * steps / (elapsed_ms / 1e3)


def run_gpu(args, rank, world, dist):
    fc = load_fc()
    dev = int(os.environ.get("LOCAL_RANK", "0"))
    n = args.n
    mesh = fc.Mesh.box(n, n, n, 1.0, 1.0, 1.0, perturb=PERTURB, seed=MESH_SEED)
    ctx = fc.Context(dev)
    ctx.set_mesh(mesh)
    nC = mesh.numCells
    b = rhs(nC)
    ctx.field_set("su", b)
    ctx.laplacian(np.ones(nC), np.zeros(mesh.numTotal), 0b1)
    nnz = 2 * mesh.numInnerFaces + nC

    def step():
        ctx.field_fill("pp", 0.0)
        r0, info, st = ctx.solve_field("iccg", "pp", "su", ITR_MAX, 0.0, TOL_REL)
        if st != 0:
            raise RuntimeError(f"ICCG status {st}")
        return info

    for _ in range(args.warmup):
        info = step()
    iters = info.itr_used
    if dist:
        dist.barrier()
    ctx.sync()
    launches0 = ctx.kernel_launches()
    solve_ms = []
    with ClockSampler(dev) as clk:
        ctx.event(0)
        for _ in range(args.steps):
            info = step()
            solve_ms.append(info.ms)
        ctx.event(1)
        elapsed = ctx.elapsed_ms()
    launches = ctx.kernel_launches() - launches0
    elapsed = max_over_ranks(dist, elapsed)
    ms_per_step = elapsed / args.steps
    value = replica_throughput(world, args.steps, elapsed)

    # end to end through the csrsolve drop-in with host buffers
    ia, ja, dg, _, _ = ctx.csr_pattern()
    a_host = ctx.field_get("a")
    pin = None
    try:
        import torch
        if torch.cuda.is_available():
            pin = lambda arr: torch.from_numpy(arr).pin_memory().numpy()  # noqa: E731
    except Exception:
        pin = None
    a_h = pin(a_host) if pin else a_host
    b_h = pin(b.copy()) if pin else b.copy()
    x_h = pin(np.zeros(nC)) if pin else np.zeros(nC)
    for _ in range(max(1, args.warmup)):
        x_h[:] = 0.0
        ctx.csrsolve_sized("iccg", nC, nnz, ia, ja, a_h, dg, x_h, b_h, ITR_MAX, 0.0, TOL_REL, "p")
    ctx.sync()
    ctx.event(0)
    for _ in range(args.steps):
        x_h[:] = 0.0
        ctx.csrsolve_sized("iccg", nC, nnz, ia, ja, a_h, dg, x_h, b_h, ITR_MAX, 0.0, TOL_REL, "p")
    ctx.event(1)
    e2e_ms = ctx.elapsed_ms() / args.steps
    h2d = a_h.nbytes + b_h.nbytes + x_h.nbytes
    d2h = x_h.nbytes

    # mixed precision (FP32 inner, FP64 refinement) to the same criterion:
    # the multicolour inner ICCG, and the natural-order one for comparison
    ctx.set_precision(fc.FC_PREC_FP64)
    step()
    x_fp64 = ctx.field_get("pp")[:nC].copy()

    def mixed_run(mode, inner_tol):
        ctx.set_precision(mode, inner_tol, 0)
        for _ in range(max(1, args.warmup)):
            mi = step()
        ctx.sync()
        ctx.event(0)
        for _ in range(args.steps):
            mi = step()
        ctx.event(1)
        ms = ctx.elapsed_ms() / args.steps
        ctx.set_precision(fc.FC_PREC_FP64)
        err = float(np.abs(ctx.field_get("pp")[:nC] - x_fp64).max() / np.abs(x_fp64).max())
        return {"value": 1e3 / ms, "unit": "p-solves/s", "ms_per_step": ms, "speedup_vs_fp64": ms_per_step / ms,
                "inner_iterations": mi.itr_used, "outer_iterations": mi.outer_iterations, "inner_tol": inner_tol,
                "max_rel_diff_vs_fp64": err}

    if args.mixed_host_loop:  # profiling: the coloured inner kernels launched from the host (more than two colours)
        ctx.set_tracing(True)
    mixed = mixed_run(fc.FC_PREC_MIXED_COLOURED, MIXED_INNER_TOL)
    ctx.set_tracing(False)
    mixed["inner_solver"] = ("FP32 ICCG, multicolour DIC (%d colours) in Eisenstat form, one persistent kernel"
                             % ctx.mixed_colours(0))
    mixed_nat = mixed_run(fc.FC_PREC_MIXED, MIXED_NATURAL_INNER_TOL)
    mixed_nat["inner_solver"] = "FP32 ICCG, natural-order DIC (the FP64 path's sweeps)"
    # precision's share of the mixed speed-up: the same multicolour inner
    # solve, refinement and stopping test in FP64
    col64 = mixed_run(fc.FC_PREC_COLOURED_FP64, MIXED_INNER_TOL)
    col64["inner_solver"] = "FP64 ICCG, the same multicolour DIC in Eisenstat form (diagnostic)"
    mixed["speedup_vs_coloured_fp64"] = col64["ms_per_step"] / mixed["ms_per_step"]

    spmv = spmv_leg(fc, ctx, nC, args.spmv_calls) if args.spmv_calls > 0 else None
    sweep = ctx.sweep_stats(0)
    peak, peak_kind = measured_peak()
    bytes_launch = iccg_bytes_per_iteration(nC, nnz) * iters
    avg_launch_ms = float(np.mean(solve_ms))
    achieved = bytes_launch / (avg_launch_ms * 1e-3) / 1e9
    # the committed ncu figure is for one 128^3 launch only
    traffic = profiled_traffic() if n == 128 else None
    if rank != 0:
        ctx.close()
        return
    # the headline keys first, the mixed-precision results right after them
    # (readers that keep only the end of a long line still see them)
    line = {"metric": METRIC, "value": value, "unit": "p-solves/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ms_per_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": workload_config(n, nC, nnz),
            "e2e": {"value": 1e3 / e2e_ms, "unit": "p-solves/s", "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h)},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": traffic,
                         "kernel": "k_iccg<double> (whole solve, one persistent launch)",
                         "peak_source": peak_kind},
            "gpu_launches": int(launches),
            "clocks": clk.summary(),
            "mixed": mixed,
            "solve": {"iterations_per_solve": iters, "parallelism": "replicas" if world > 1 else "single GPU",
                      "sweep_tiles": int(sweep["tiles"]), "sweep_levels": int(sweep["levels"]),
                      "sweep_est_us": round(sweep["est_sweep_us"], 1)},
            "mixed_natural_order": mixed_nat,
            "coloured_fp64": col64}
    if spmv:
        line["spmv"] = spmv
    ctx.close()
    if not args.no_cpu:
        line["cpu_baseline"] = cpu_baseline(ia, ja, a_host, dg, b)
    if args.simple_n > 0:
        line["simple"] = simple_block(fc, args, dev, not args.no_cpu, args.simple_n)
    if args.grad_n > 0:
        line["gradients"] = gradient_block(fc, args, dev)
    if args.adjoint_n > 0:
        line["adjoint"] = adjoint_block(fc, args, dev)
    if args.batch_count > 0:
        line["batch"] = batch_block(fc, args, dev)
    if args.piso_n > 0:
        line["piso"] = piso_block(fc, args, dev, not args.no_cpu)
    if args.turb_n > 0:
        line["turbulence"] = turbulence_block(fc, args, dev, not args.no_cpu)
    if args.simple_tet_n > 0:
        # C5: 6 tets per perturbed hex, Re = 400, LSQ gradients, boundedLinearUpwind.  With the cavity
        # input's urfU 0.8 / urfP 0.3 the SIMPLE iteration diverges on this mesh (the oracle too, at
        # 40^3 x 6 tets); 0.6 / 0.2 converges
        line["simple_tets"] = simple_block(fc, args, dev, not args.no_cpu, args.simple_tet_n, PERTURB, cpu_skip=0,
                                           tets=True, viscos=1.0 / 400.0, scheme=19, grad=1,
                                           iters=args.simple_tet_iters, cpu_iters=1, urf=(0.6, 0.2))
    if args.simple_big_n > 0:
        line["simple_perturbed"] = simple_block(fc, args, dev, not args.no_cpu, args.simple_big_n, PERTURB,
                                                cpu_skip=args.simple_big_cpu_skip, momentum_batch=True,
                                                iters=args.simple_big_iters, skip=args.simple_big_skip)
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--n", "--cells-per-side", dest="n", type=int, default=128, help="cells per side of the cube")
    ap.add_argument("--ref-warmup-iters", type=int, default=10,
                    help="ICCG iterations of each warm-up step of the reference arm")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--spmv-calls", type=int, default=20, help="timed fc_spmv calls on device arrays (0: skip)")
    ap.add_argument("--mixed-host-loop", action="store_true",
                    help="launch the multicolour inner kernels of more than two colours from the host "
                         "(visible to profilers)")
    ap.add_argument("--simple-n", type=int, default=64, help="cells per side of the SIMPLE cavity (0: skip)")
    ap.add_argument("--simple-big-n", type=int, default=128,
                    help="cells per side of the SIMPLE cavity on the perturbed mesh (0: skip)")
    ap.add_argument("--simple-big-cpu-skip", type=int, default=2, help="untimed oracle iterations there")
    ap.add_argument("--simple-tet-n", type=int, default=0,
                    help="hexes per side of the tetrahedral SIMPLE cavity, 6 tets each (0: skip; 100 = 6M cells)")
    ap.add_argument("--simple-tet-iters", type=int, default=100, help="timed SIMPLE iterations there")
    ap.add_argument("--grad-n", type=int, default=128, help="cells per side of the gradient-kernel leg (0: skip)")
    ap.add_argument("--grad-calls", type=int, default=20, help="timed fc_grad calls per scheme there")
    ap.add_argument("--adjoint-n", type=int, default=96, help="cells per side of the adjoint case (0: skip)")
    ap.add_argument("--adjoint-fd-dirs", type=int, default=32, help="directions of the finite-difference check")
    ap.add_argument("--momentum-calls", type=int, default=5, help="timed calcuvw calls of the C3a leg")
    ap.add_argument("--piso-n", type=int, default=64, help="cells per side of the PISO leg (0: skip)")
    ap.add_argument("--turb-n", type=int, default=128, help="cells per side of the k-omega SST leg (0: skip)")
    ap.add_argument("--turb-calls", type=int, default=5, help="timed fc_kw_sst calls there")
    ap.add_argument("--piso-steps", type=int, default=10, help="timed PISO time steps")
    ap.add_argument("--batch-count", type=int, default=64, help="problems of the batched leg (0: skip)")
    ap.add_argument("--batch-tol", type=float, default=BATCH_TOL, help="relative L1 tolerance there")
    ap.add_argument("--batch-inner-tol", type=float, default=BATCH_INNER_TOL, help="FP32 inner tolerance there")
    ap.add_argument("--batch-inner-itmax", type=int, default=BATCH_INNER_ITMAX, help="FP32 inner iteration cap there")
    ap.add_argument("--batch-reps", type=int, default=2, help="timed repetitions of each batched leg")
    ap.add_argument("--batch-tune-rounds", type=int, default=2, help="autotuner plans tried")
    ap.add_argument("--batch-cpu-seconds", type=float, default=10.0, help="oracle time of the CPU estimate")
    ap.add_argument("--simple-iters", type=int, default=200,
                    help="timed SIMPLE iterations of the 64^3 cavity (the configuration's 200 outer iterations)")
    ap.add_argument("--simple-skip", type=int, default=0, help="untimed SIMPLE iterations before them")
    ap.add_argument("--simple-big-iters", type=int, default=20, help="timed SIMPLE iterations of the 128^3 leg")
    ap.add_argument("--simple-big-skip", type=int, default=10, help="untimed SIMPLE iterations before them")
    ap.add_argument("--simple-cpu-iters", type=int, default=3, help="oracle SIMPLE iterations timed")
    args = ap.parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("gloo")
    if args.impl == "reference":
        run_reference(args, rank, world)
    else:
        run_gpu(args, rank, world, dist)
    if dist:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
