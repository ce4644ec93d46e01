#!/usr/bin/env python
"""Benchmark: milliseconds per 60k-DOF plate solve at FP64-checked error 1e-6.

One step = one complete solve of the plate_q4_141 workload (141x141 Q4
Mindlin, 60,492 DOF, seeded synthetic loads and column supports) through
pg_plan_solve_device: the persistent PCG launch with its result readback,
inputs resident in HBM (the plan's element stiffness, block-Jacobi and
coarse set-up ran in the warm-up and is cached).  Seven methods are timed
(FP64 / mixed precision x block Jacobi / two-level x Chebyshev smoother);
``value`` is the fastest whose FP64-checked error is <= 1e-6, in ms per
solve for the whole job (lower is better).  ``e2e`` is the same through
the public C ABI (pg_solve) from host buffers, copies included;
``first_solve_new_mesh_ms`` a first pg_solve in a new context (the plan's
set-up included; the median of three, each in its own new context;
``first_solve_new_mesh_phases`` splits that run as the library times it:
partition plan, coarse space, eigenvalue estimate, device set-up and
solve).  L2 is flushed (256 MiB write) between timed steps; each
step is timed with CUDA events on the solver's stream.  ``roofline``
compares the PCG kernel's algorithmic bytes per second with the measured
HBM copy peak and with an in-run L2-resident copy.

Every variant's FP64 error is checked on the plate's own load and 16
seeded random-field loads; only a variant whose largest error is <= 1e-6
can be the headline.

The whole line goes to stderr; stdout gets it with its sections cut to
their main numbers (summary), so that it survives in the tail of a log.
Further sections of the line: ``learned`` (the learned two-level
preconditioner: flexible PCG with the trained U-Net, one CUDA graph per
solve; timed like the variants, checked on the same loads, evaluated on
512 held-out loads, compared with the same loop without the network, and
the network's forward pass against the BF16 tensor-core peak),
``load_cases`` (four loads of the plate through pg_solve_load_cases
against the same loads one by one), ``other_configs`` (plate_q4_32,
plate_dkt_200, the unstructured plate_holes_dkt and plate_q4_400, which
runs on the global-memory path; four methods each), ``batch`` (a 256-plate
uneven batch, Q4 and DKT, sides 16-256, team-size target autotuned, four
methods, the fastest that meets the error bar reported; errors on the 5
largest plates and 5% of the others against sparse LU and on every plate
against an FP64 1e-12 solve) and ``cpu_baseline`` (the reference-precision
CPU solver, one core).  --learned 0, --cases 0, --other-configs 0,
--batch 0 skip sections.

Multi-GPU: a single plate does not shard (the solve is bound by the
latency of the exchange between blocks), so --gpus N runs N independent
replicas, one per rank, and ``value`` = max-over-ranks time / (N * steps);
the batch is sharded across the ranks by estimated cost.

--impl reference times the reference's CPU algorithm (the oracle's
restatement of solvePCG + applyGlobalK in reference precision; the
TypeScript original cannot run here) on the host.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(ROOT, "gpu-gauntlet_b200"))

METRIC = "ms per 60k-DOF plate solve at 1e-6 FP64-checked error: learned/mixed vs plain PCG"
FALLBACK_HBM_GBS = 6650.0
# name -> (precision, preconditioner, smoother); "fp64" is the plain
# method.  Each runs at the residual tolerance of TOLERANCES (the two-level
# iterates are closer to the solution at equal residual), and the bench
# checks the error of every variant against the FP64 truth on the plate's
# own load and ACCURACY_LOADS seeded random-field loads.
VARIANTS = {"fp64": ("fp64", "bj", "bj"), "mixed": ("mixed", "bj", "bj"),
            "mixed_cheb": ("mixed", "bj", "cheb"),
            "fp64_two_level": ("fp64", "tl", "bj"), "mixed_two_level": ("mixed", "tl", "bj"),
            "fp64_two_level_cheb": ("fp64", "tl", "cheb"),
            "mixed_two_level_cheb": ("mixed", "tl", "cheb")}
# residual tolerances (block Jacobi, two-level) that keep the FP64 error at
# or below 1e-6 on the plate's own load and on seeded random-field loads:
# plate_q4_141 two-level 3e-6 (at 5e-6 a seeded load reached 1.35e-6; at
# 3e-6 the worst of 17 loads is about 6e-7 in a CPU model of the FP64
# method); the reference's DKT formulation needs a tighter residual for the
# same error (1.15e-6 at 1e-6, 1.6e-7 at 1e-7); plate_q4_32 runs at its
# configured rtol 1e-8
TOLERANCES = {"plate_q4_141": (1e-6, 3e-6), "plate_dkt_200": (1e-7, 1e-7), "plate_q4_32": (1e-8, 1e-8),
              # the global-memory path (plate too large for shared memory); its
              # FP64 error at this stop is checked by the GPU tests (sparse LU of
              # 482,403 DOF takes too long for the benchmark)
              "plate_q4_400": (1e-8, 1e-8),
              # FP64 error about 2.5 x the relative residual on this mesh
              "plate_holes_dkt": (2e-7, 2e-7)}
WORKLOAD_DATA = {
    "plate_q4_141": "synthetic (seeded plate_q4_141: 5 kPa + 32 point loads, 16 columns)",
    "plate_q4_32": "synthetic (seeded plate_q4_32: 1 kPa + 4 point loads, clamped)",
    "plate_dkt_200": "synthetic (seeded plate_dkt_200: jittered DKT mesh, GRF thickness, "
                     "3 kPa, clamped)",
    "plate_q4_400": "synthetic (seeded plate_q4_400: 400x400 Q4, 482,403 DOF, 5 kPa + 32 point loads, "
                    "16 columns)",
    "plate_holes_dkt": "synthetic (seeded plate_holes_dkt: Delaunay DKT plate with two holes, "
                       "shuffled node numbers, 4 kPa + 2 point loads, clamped outer edges)",
}
# algorithmic vector words per DOF and iteration (the minimal fused PCG
# schedule: K.p 2, x 3, r 3, block Jacobi 5, p 3); the Chebyshev smoother
# adds its K.t (2) and a second block-Jacobi product (3)
WORDS = {"bj": 16, "cheb": 21}
# seeded random-field loads (Gaussian random field pressure + 0-16 point
# loads) on which every variant's FP64 error is checked besides the plate's
# own load; a variant is eligible for the headline only when its largest
# error over all of them is <= 1e-6
ACCURACY_LOADS = 16
ACCURACY_SEED = 77


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", choices=["plategpu", "reference"], default="plategpu")
    ap.add_argument("--workload", default="plate_q4_141")
    ap.add_argument("--variants", default=",".join(VARIANTS),
                    help="comma-separated subset of " + ",".join(VARIANTS))
    ap.add_argument("--tol-bj", type=float, default=None,
                    help="||r||/||b|| tolerance with block Jacobi (default per workload)")
    ap.add_argument("--tol-tl", type=float, default=None,
                    help="||r||/||b|| tolerance with the two-level preconditioner (default per workload)")
    ap.add_argument("--ctas", type=int, default=0)
    ap.add_argument("--threads", type=int, default=0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--e2e-steps", type=int, default=0, help="0 = same as --steps")
    ap.add_argument("--batch", type=int, default=256,
                    help="plates of the uneven batch measured beside the headline (0 = skip)")
    ap.add_argument("--batch-steps", type=int, default=3)
    ap.add_argument("--batch-fp64", type=int, default=1,
                    help="1: also time the batch in plain FP64 (two-level, and block Jacobi)")
    ap.add_argument("--cases", type=int, default=4,
                    help="load cases of the workload plate solved together (0 = skip)")
    ap.add_argument("--cases-steps", type=int, default=5)
    ap.add_argument("--learned", type=int, default=1,
                    help="1: also time the learned two-level preconditioner (needs its weight file)")
    ap.add_argument("--learned-held-out", type=int, default=512,
                    help="held-out random-field loads evaluated with the learned preconditioner")
    ap.add_argument("--other-configs", type=int, default=1,
                    help="1: also time the other single-plate configs (plate_q4_32, plate_dkt_200, "
                         "plate_holes_dkt)")
    args = ap.parse_args()
    bj, tl = TOLERANCES.get(args.workload, (1e-6, 1e-6))
    args.tol_bj = bj if args.tol_bj is None else args.tol_bj
    args.tol_tl = tl if args.tol_tl is None else args.tol_tl
    return args


# ---------------------------------------------------------------------------
# distributed plumbing (replicas)
# ---------------------------------------------------------------------------

def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist

        if torch.cuda.is_available():
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                    device_id=torch.device("cuda", local))
        else:  # host-only runs of the plumbing (tests)
            dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=120))
    return world, rank, local


def barrier(world):
    if world > 1:
        import torch.distributed as dist

        dist.barrier()


def max_over_ranks(world, value, local):
    if world == 1:
        return value
    import torch
    import torch.distributed as dist

    dev = f"cuda:{local}" if torch.cuda.is_available() else "cpu"
    t = torch.tensor([value], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------

class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "100"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        time.sleep(0.4)

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, power, reasons = [], [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
                power.append(float(parts[3]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        os.unlink(self.path)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "power_w_max": max(power) if power else None,
                "samples": len(sm), "reasons": sorted(reasons)}


def hbm_peak():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs, copy burst)"
    except (OSError, KeyError, ValueError):
        return FALLBACK_HBM_GBS, "fallback (6.65 TB/s earlier measurement on this pool)"


def l2_copy_peak(local):
    """Copy bandwidth (read + write bytes per second, GB/s) with a working
    set of 2 x 32 MB, which stays in L2, measured in this run with CUDA
    events.  Smaller copies are bound by launch latency and 2 x 48 MB
    already spills to HBM (measured: 6.9, 8.2 and 6.1 TB/s at 2 x 24, 32 and
    48 MB), so this is a lower bound of the L2 roof against which the
    persistent kernel is also compared (its vectors live in shared memory
    and L2)."""
    import torch

    a = torch.ones(8 << 20, dtype=torch.float32, device=f"cuda:{local}")
    b = torch.empty_like(a)
    for _ in range(10):
        b.copy_(a)
    s_, e_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    s_.record()
    reps = 400
    for _ in range(reps):
        b.copy_(a)
    e_.record()
    torch.cuda.synchronize()
    ms = s_.elapsed_time(e_)
    return 2.0 * a.numel() * 4 * reps / (ms * 1e-3) / 1e9


def ncu_traffic(kernel_tag, workload):
    """DRAM bytes per launch from the committed ncu summary, if present."""
    p = os.path.join(ROOT, "profiles", f"{kernel_tag}_{workload}.txt")
    try:
        for line in open(p):
            if line.startswith("dram_bytes_per_launch:"):
                return float(line.split(":", 1)[1].split()[0])
    except OSError:
        pass
    return None


# ---------------------------------------------------------------------------
# checker (the oracle, test infrastructure) -- cpu_baseline leg only
# ---------------------------------------------------------------------------

def oracle_checks(wl, want_baseline=True):
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import numpy as np
    import oracle as O

    m, mat = wl.mesh, wl.material
    npe = m.nodesPerElement
    F = wl.F.astype(np.float64)
    ke64 = O.all_ke(m.nodes, m.elements, npe, mat.E, mat.nu, mat.t, elem_t=mat.elem_t,
                    mode=O.FP64)
    solve = O.truth_factor(m.nodeCount, m.elements, npe, ke64, wl.cons_mask)
    xs, rel = solve(F)
    out = {"truth": xs, "A": solve.A, "solve": solve}
    if want_baseline:
        keR = O.all_ke(m.nodes, m.elements, npe, mat.E, mat.nu, mat.t, elem_t=mat.elem_t,
                       mode=O.REF)
        offs, flat = wl.coloring.flat()
        t0 = time.perf_counter()
        bd = O.invert_block_diag(O.block_diag(m.nodeCount, m.elements, npe, keR, O.REF),
                                 wl.cons_mask, O.REF)
        xr, it, res, conv = O.solve_pcg(m.nodeCount, m.elements, npe, keR, offs, flat,
                                        wl.cons_mask, bd, F, 1e-6, 20000, O.REF)
        ms = (time.perf_counter() - t0) * 1e3
        out.update(ref_x=xr, ref_iters=it, ref_conv=conv, ref_ms=ms)
    return out


def accuracy(x, chk):
    import numpy as np

    xs, A = chk["truth"], chk["A"]
    e = x - xs
    res = {"rel_l2_vs_fp64_truth": float(np.linalg.norm(e) / np.linalg.norm(xs)),
           "energy_norm_rel": float(np.sqrt(abs(e @ (A @ e)) / abs(xs @ (A @ xs)))),
           "max_w_rel_vs_fp64_truth": None, "max_w_rel_vs_reference_cpu": None}
    w, ws = x[0::3], xs[0::3]
    mw, mws = w[np.argmax(np.abs(w))], ws[np.argmax(np.abs(ws))]
    res["max_w_rel_vs_fp64_truth"] = float(abs(mw - mws) / abs(mws))
    if "ref_x" in chk:
        wr = chk["ref_x"][0::3]
        mwr = wr[np.argmax(np.abs(wr))]
        res["max_w_rel_vs_reference_cpu"] = float(abs(mw - mwr) / abs(mwr))
    return res


# ---------------------------------------------------------------------------
# arms
# ---------------------------------------------------------------------------

def bench_config(wl, args):
    """The workload description that both arms print as `config` (the
    method each arm ran is reported beside it, not in it)."""
    return {"workload": args.workload, "dof": wl.n_dof, "elements": wl.mesh.elementCount,
            "accuracy": "FP64 relative L2 error <= 1e-6 vs the FP64 truth",
            "l2": "GPU arm: flushed between steps (256 MiB write)",
            "parallelism": "replicas"}


def run_reference(args, world, rank):
    """The reference CPU algorithm (oracle port, reference precision): each
    step is one complete solve as solvePlate runs it -- element matrices,
    block diagonal and its inversion, then PCG to the reference's tolerance
    1e-6 with the iteration cap raised so that it converges."""
    if rank != 0:
        return
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import numpy as np
    import oracle as O
    from plategpu import workloads

    wl = workloads.WORKLOADS[args.workload]()
    m, mat = wl.mesh, wl.material
    npe = m.nodesPerElement
    F = wl.F.astype(np.float64)
    offs, flat = wl.coloring.flat()

    def solve(maxit, tol):
        ke = O.all_ke(m.nodes, m.elements, npe, mat.E, mat.nu, mat.t, elem_t=mat.elem_t,
                      mode=O.REF)
        bd = O.invert_block_diag(O.block_diag(m.nodeCount, m.elements, npe, ke, O.REF),
                                 wl.cons_mask, O.REF)
        return O.solve_pcg(m.nodeCount, m.elements, npe, ke, offs, flat, wl.cons_mask, bd, F,
                           tol, maxit, O.REF)

    for _ in range(args.warmup):
        solve(20000, 1e-6)
    times, full_iters, conv = [], 0, False
    for _ in range(args.steps):
        t0 = time.perf_counter()
        _x, full_iters, _r, conv = solve(20000, 1e-6)
        times.append((time.perf_counter() - t0) * 1e3)
    value = statistics.mean(times)
    sample = (f"one complete reference-precision solve of {args.workload} per step "
              f"(set-up once + {full_iters} PCG iterations to tolerance 1e-6, "
              f"converged={conv}) by the C restatement of solvePlate/solvePCG/applyGlobalK; "
              "single thread (the reference's JavaScript solver runs on one thread)")
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "ms",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": value, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32 storage / f64 arithmetic",
            "data": WORKLOAD_DATA.get(args.workload, "synthetic (seeded workload)"),
            "config": bench_config(wl, args), "iterations": full_iters,
            "cpu_baseline": {"value": value, "unit": "ms", "cores": 1, "kind": "port",
                             "sample": sample},
            "e2e": {"value": value, "unit": "ms", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def describe_preconditioner(v, coarse_dim):
    sm = ("Chebyshev smoother (degree 2 in D^-1 K, 2-ring halo)" if v[2] == "cheb"
          else "block Jacobi")
    return (f"two-level ({sm} + coarse correction, {coarse_dim} coarse DOFs)" if v[1] == "tl"
            else sm)


def variant_options(args, name):
    from plategpu import _lib

    precision, pre, smoother = VARIANTS[name]
    prec = _lib.PG_PREC_FP64 if precision == "fp64" else _lib.PG_PREC_MIXED
    tl = pre == "tl"
    return _lib.make_options(
        tolerance=args.tol_tl if tl else args.tol_bj, max_iterations=20000, precision=prec,
        stop_rule=_lib.PG_STOP_RELATIVE, ctas=args.ctas, threads=args.threads,
        preconditioner=_lib.PG_PRECOND_TWO_LEVEL if tl else _lib.PG_PRECOND_BLOCK_JACOBI,
        smoother=_lib.PG_SMOOTHER_CHEBYSHEV if smoother == "cheb" else _lib.PG_SMOOTHER_BLOCK_JACOBI,
        # mixed with the Chebyshev smoother: FP64 residual replacement every
        # two decades of the FP32 residual (3 instead of 6 on plate_q4_141 at
        # the same error; without the smoother it costs iterations)
        reliable_delta=0.01 if (prec == _lib.PG_PREC_MIXED and smoother == "cheb") else 0.0)


def time_variant(args, world, local, ctx, prob, name, stream, F_dev, x_dev, flush, extra_F=None):
    """Warm-up + timed device-resident solves of one variant; then, untimed,
    the loads of extra_F (device [k, n] float) with the same plan, whose
    solutions are returned as "x_extra"."""
    import torch

    opts = variant_options(args, name)
    plan = ctx.plan(prob, opts)
    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            plan.solve_device(opts, F_dev.data_ptr(), x_dev.data_ptr())
        starts = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
        ends = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
        infos = []
        barrier(world)
        torch.cuda.synchronize()
        for k in range(args.steps):
            flush.fill_(k & 0xFF)
            starts[k].record(stream)
            infos.append(plan.solve_device(opts, F_dev.data_ptr(), x_dev.data_ptr()))
            ends[k].record(stream)
        torch.cuda.synchronize()
        barrier(world)
    step_ms = [s_.elapsed_time(e_) for s_, e_ in zip(starts, ends)]
    total = max_over_ranks(world, sum(step_ms), local)
    x_main = x_dev.cpu().numpy().copy()
    x_extra = []
    if extra_F is not None:
        with torch.cuda.stream(stream):
            for k in range(extra_F.shape[0]):
                plan.solve_device(opts, extra_F[k].data_ptr(), x_dev.data_ptr())
                x_extra.append(x_dev.cpu().numpy().copy())
    plan.close()
    return {"opts": opts, "value": total / (world * args.steps), "step_ms": step_ms,
            "kernel_ms": statistics.mean(i.solve_ms for i in infos),
            "setup_ms": statistics.mean(i.setup_ms for i in infos),
            "iterations": infos[-1].iterations, "reductions": infos[-1].reductions,
            "tolerance": opts.tolerance, "coarse_dim": infos[-1].coarse_dim,
            "reliable_updates": infos[-1].reliable_updates,
            "true_rel_residual": infos[-1].true_rel_residual,
            "ctas": infos[-1].ctas, "threads": infos[-1].threads,
            "global_path": infos[-1].global_path,
            "x": x_main, "x_extra": x_extra}


def run_plategpu(args, world, rank, local):
    import numpy as np
    import torch

    from plategpu import _lib, workloads

    torch.cuda.set_device(local)
    wl = workloads.WORKLOADS[args.workload]()
    n = wl.n_dof
    ctx = _lib.Context(local)
    stream = torch.cuda.Stream(device=local)
    ctx.set_stream(stream.cuda_stream)
    prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
    F_dev = torch.from_numpy(wl.F).to(f"cuda:{local}")
    x_dev = torch.zeros(n, dtype=torch.float64, device=f"cuda:{local}")
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=f"cuda:{local}")
    variants = [v for v in args.variants.split(",") if v]
    for v in variants:
        if v not in VARIANTS:
            raise SystemExit(f"unknown variant {v!r}")

    check = rank == 0 and world == 1 and not args.no_cpu_baseline
    extra_F = None
    if check and args.workload == "plate_q4_141":
        extra_F = torch.from_numpy(
            workloads.random_field_loads(wl, ACCURACY_LOADS, ACCURACY_SEED)).to(f"cuda:{local}")

    sampler = ClockSampler(local) if rank == 0 else None
    if sampler:
        sampler.start()
    res = {v: time_variant(args, world, local, ctx, prob, v, stream, F_dev, x_dev, flush, extra_F)
           for v in variants}
    clocks = sampler.stop() if sampler else None

    chk = None
    if check:
        chk = oracle_checks(wl, want_baseline=True)
        extra_truth = ([chk["solve"](f)[0] for f in extra_F.cpu().numpy()]
                       if extra_F is not None else [])
        for v in variants:
            res[v]["accuracy"] = accuracy(res[v]["x"], chk)
            errs = [res[v]["accuracy"]["rel_l2_vs_fp64_truth"]] + [
                float(np.linalg.norm(x - xt) / np.linalg.norm(xt))
                for x, xt in zip(res[v]["x_extra"], extra_truth)]
            res[v]["accuracy"]["loads"] = {
                "count": len(errs), "rel_l2_max": max(errs),
                "rel_l2_p50": float(np.percentile(errs, 50)),
                "rel_l2_p99": float(np.percentile(errs, 99)),
                "loads": (f"the plate's own load + {len(errs) - 1} seeded random-field loads "
                          f"(seed {ACCURACY_SEED})")}
    # headline: the fastest variant whose FP64-checked error meets 1e-6 on
    # every load checked (without the checker, the fastest variant whose
    # true residual met the tolerance)
    def meets(v):
        acc = res[v].get("accuracy")
        if acc is not None:
            return acc["loads"]["rel_l2_max"] <= 1e-6
        return res[v]["true_rel_residual"] <= res[v]["tolerance"]
    ok = [v for v in variants if meets(v)] or variants
    head = min(ok, key=lambda v: res[v]["value"])
    H = res[head]

    # e2e through the C ABI from host buffers (pg_solve), headline variant
    e2e_steps = args.e2e_steps or args.steps
    rng = np.random.default_rng(1234)
    loads = [(wl.F * np.float32(1.0 + 0.1 * rng.random())).astype(np.float32)
             for _ in range(min(e2e_steps, 16))]
    for k in range(2):
        prob.set_F(loads[k % len(loads)])
        ctx.solve(prob, H["opts"])
    barrier(world)
    e2e = []
    for k in range(e2e_steps):
        prob.set_F(loads[k % len(loads)])
        t0 = time.perf_counter()
        ctx.solve(prob, H["opts"])
        e2e.append((time.perf_counter() - t0) * 1e3)
    barrier(world)
    e2e_value = max_over_ranks(world, sum(e2e), local) / (world * e2e_steps)
    # a first solve of the plate in a new context: partition, element
    # matrices, coarse space and eigenvalue estimate, then the solve
    # (three times, each in its own new context; the median is reported with
    # its one-time steps as the library times them: host wall time, the
    # device set-up and solve by CUDA events)
    prob.set_F(wl.F)
    colds = []
    for _ in range(3):
        cold_ctx = _lib.Context(local)
        t0 = time.perf_counter()
        _xc, cold_info = cold_ctx.solve(prob, H["opts"])
        ms_c = max_over_ranks(world, (time.perf_counter() - t0) * 1e3, local)
        cold_ctx.close()
        colds.append((ms_c, {"partition_plan_ms": cold_info.plan_ms, "coarse_space_ms": cold_info.coarse_ms,
                             "eigenvalue_estimate_ms": cold_info.eigen_ms, "device_setup_ms": cold_info.setup_ms,
                             "device_solve_ms": cold_info.solve_ms}))
    colds_sorted = sorted(colds, key=lambda c: c[0])
    cold_ms, cold_phases = colds_sorted[1]
    cold_phases = dict(cold_phases, all_runs_ms=[c[0] for c in colds])
    # the same cold path in two steps: the plan (host partition, device
    # copies) and its first device solve (element matrices, block inverses,
    # coarse space, eigenvalue estimate, then the solve)
    cold_ctx = _lib.Context(local)
    cold_ctx.set_stream(stream.cuda_stream)
    t0 = time.perf_counter()
    cold_plan = cold_ctx.plan(prob, H["opts"])
    t1 = time.perf_counter()
    with torch.cuda.stream(stream):
        cinfo = cold_plan.solve_device(H["opts"], F_dev.data_ptr(), x_dev.data_ptr())
    t2 = time.perf_counter()
    cold_split = {"plan_ms": (t1 - t0) * 1e3, "first_solve_ms": (t2 - t1) * 1e3,
                  "first_solve_device_setup_ms": cinfo.setup_ms, "first_solve_device_solve_ms": cinfo.solve_ms}
    cold_plan.close()
    cold_ctx.close()
    cases = (cases_bench(args, ctx, wl, prob, H, head, chk is not None, world, local)
             if args.cases > 0 else None)
    lrn = (learned_bench(args, ctx, stream, flush, local, wl, chk, extra_F)
           if args.learned and rank == 0 else None)
    others = (other_configs_bench(args, ctx, stream, flush, world, local, chk is not None)
              if args.other_configs else None)
    # every rank takes part in the batch (its share of the plates)
    batch = batch_bench(args, ctx, chk is not None, world, rank, local) if args.batch > 0 else None

    if rank != 0:
        ctx.close()
        return
    # roofline of the dominant kernel: algorithmic bytes per launch
    # (16 vector words per DOF per iteration; 8-byte words in FP64, 4-byte
    # words for the FP32 inner iterations)
    word = 8 if VARIANTS[head][0] == "fp64" else 4
    iters = H["iterations"]
    alg_bytes = float(WORDS[VARIANTS[head][2]]) * n * word * iters
    peak, peak_src = hbm_peak()
    achieved = alg_bytes / (H["kernel_ms"] * 1e-3) / 1e9
    l2_peak = l2_copy_peak(local)
    kernel_tag = "pcg_" + head
    line = {
        "metric": METRIC, "value": H["value"], "unit": "ms", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": statistics.mean(H["step_ms"]),
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if VARIANTS[head][0] == "fp64" else "f32 inner / f64 refinement",
        "data": WORKLOAD_DATA.get(args.workload, "synthetic (seeded workload)"),
        "config": bench_config(wl, args),
        "method": {"name": head,
                   "preconditioner": describe_preconditioner(VARIANTS[head], H["coarse_dim"]),
                   "stop": f"||r||/||b|| < {H['tolerance']:g}", "ctas": H["ctas"],
                   "threads": H["threads"], "replicas": world},
        "iterations": iters,
        "kernel_ms": H["kernel_ms"], "setup_ms": H["setup_ms"],
        "us_per_iteration": H["kernel_ms"] * 1e3 / max(iters, 1),
        "variants": {v: {k: res[v][k] for k in ("value", "kernel_ms", "setup_ms", "iterations",
                                               "reductions", "reliable_updates", "tolerance",
                                               "true_rel_residual", "coarse_dim")}
                     | {"accuracy": res[v].get("accuracy")} for v in variants},
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "traffic": ncu_traffic(kernel_tag, args.workload),
                     "kernel": f"{kernel_tag}_kernel", "peak_source": peak_src,
                     "algorithmic_bytes_per_launch": alg_bytes,
                     "l2": {"peak": l2_peak, "frac": achieved / l2_peak, "unit": "GB/s",
                            "peak_source": ("copy with a 2 x 32 MB working set, L2-resident, measured "
                                            "in this run (a lower bound of the L2 bandwidth)")}},
        "e2e": {"value": e2e_value, "unit": "ms", "h2d_bytes_per_step": 4 * n,
                "d2h_bytes_per_step": 8 * n + 64},
        "first_solve_new_mesh_ms": cold_ms,
        "first_solve_new_mesh_split": cold_split,
        "first_solve_new_mesh_phases": cold_phases,
        # one persistent PCG launch per timed solve: the plan's set-up kernels
        # (element matrices, block inverses, task blocks) ran in the warm-up
        "gpu_launches": args.steps,
        "clocks": clocks,
        "accuracy": H.get("accuracy"),
    }
    if cases is not None:
        line["load_cases"] = cases
    if lrn is not None:
        line["learned"] = lrn
    if others:
        line["other_configs"] = others
    if batch is not None:
        line["batch"] = batch
    if chk is not None:
        line["cpu_baseline"] = {
            "value": chk["ref_ms"], "unit": "ms", "cores": 1, "kind": "port",
            "sample": (f"one full reference-precision solve of {args.workload} "
                       f"({chk['ref_iters']} iterations, tol 1e-6) by the C restatement "
                       "of solvePCG/applyGlobalK, single thread")}
    else:
        line["cpu_baseline"] = None
    print(json.dumps(line), file=sys.stderr, flush=True)
    print(json.dumps(summary(line), separators=(",", ":")), flush=True)
    ctx.close()


# relative FP64 true residual of the learned flexible PCG and of the same
# loop without the network: at 1e-6 one of the 512 held-out loads ended at
# 1.02e-6 FP64 error; 5e-7 keeps every load under the 1e-6 bar
LEARNED_TOL = 5e-7


SECTIONS = ("config", "variants", "load_cases", "learned", "other_configs", "batch", "first_solve_new_mesh_split",
            "first_solve_new_mesh_phases", "roofline", "method", "accuracy", "cpu_baseline")


def pick(d, *keys):
    """Those of `keys` that d has (d may be None), floats to five digits."""
    return {k: float(f"{d[k]:.5g}") if isinstance(d[k], float) else d[k] for k in keys if d and k in d}


def summary(line):
    """The line with its sections cut to their main numbers, under 2.5 KB, which survives in the tail of a log; the
    whole of it goes to stderr."""
    out = {k: v for k, v in line.items() if k not in SECTIONS}
    out["config"] = {k: v for k, v in line["config"].items() if not (isinstance(v, str) and len(v) > 60)}
    out["variants_ms"] = {v: float(f"{r['value']:.5g}") for v, r in line.get("variants", {}).items()}
    out["method"] = line["method"]["name"]
    out["rel_l2_max"] = ((line.get("accuracy") or {}).get("loads") or {}).get("rel_l2_max")
    out["roofline"] = pick(line.get("roofline"), "bound", "achieved", "peak", "unit", "frac")
    for name, keys in (("load_cases", ("cases", "device_ms_per_case", "e2e_ms_per_case", "speedup_e2e")),
                       ("learned", ("value", "iterations", "us_per_iteration")),
                       ("batch", ("method", "batch_ms", "solves_per_s", "plate_ms_p99", "max_rel_l2_vs_fp64_truth")),
                       ("cpu_baseline", ("value", "unit", "cores", "kind"))):
        out[name] = pick(line.get(name), *keys) or None
    out["other_configs_ms"] = {n: pick(r, "best_ms").get("best_ms") for n, r in (line.get("other_configs") or {}).items()}
    return out


def learned_bench(args, ctx, stream, flush, local, wl, chk, extra_F):
    """The learned two-level preconditioner on the workload plate: the U-Net
    trained by ``python -m plategpu.learned train`` (its weight file ships
    with the package) as the coarse correction inside flexible PCG, one
    CUDA graph launch per solve.  Timed like the headline variants
    (device-resident loads, L2 flushed between steps); FP64 error on the same
    loads as the variants when the checker runs; held-out random-field loads
    (seeded differently from the training loads) for iterations and time;
    the same flexible PCG without the network (smoothing steps only, and
    plain block Jacobi) for the gain; and the network's forward pass alone
    (batch 1 and 32) against the BF16 tensor-core peak."""
    import numpy as np
    import torch

    from plategpu import _lib, learned

    path = learned.DEFAULT_WEIGHTS
    if args.workload != "plate_q4_141" or not os.path.exists(path):
        return {"unavailable": f"no trained network for {args.workload} ({os.path.basename(path)} absent)"}
    ls = learned.LearnedSolver(ctx, wl, weights=path)
    meta = {}
    try:
        meta = learned.load_weights(ls.net, path)
        n = wl.n_dof
        F_dev = torch.from_numpy(wl.F).to(f"cuda:{local}")
        x_dev = torch.zeros(n, dtype=torch.float64, device=f"cuda:{local}")
        opts = learned.solve_options(LEARNED_TOL, max_iterations=2000)
        steps = max(3, args.steps // 2)
        with torch.cuda.stream(stream):
            for _ in range(args.warmup):
                ls.learned.solve_device(opts, F_dev.data_ptr(), x_dev.data_ptr())
            ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
                  for _ in range(steps)]
            infos = []
            torch.cuda.synchronize()
            for k in range(steps):
                flush.fill_(k & 0xFF)
                ev[k][0].record(stream)
                infos.append(ls.learned.solve_device(opts, F_dev.data_ptr(), x_dev.data_ptr()))
                ev[k][1].record(stream)
            torch.cuda.synchronize()
        ms = [a.elapsed_time(b) for a, b in ev]
        info, st = infos[-1]
        out = {"method": "flexible PCG (Polak-Ribiere), two-level: block-Jacobi smoothing + U-Net "
                         "correction (BF16 tensor cores), FP64 true-residual stop",
               "stop": f"||F - K x|| / ||F|| < {LEARNED_TOL:g} (FP64)",
               "value": statistics.mean(ms), "graph_ms": statistics.mean(i[0].solve_ms for i in infos),
               "iterations": int(info.iterations), "network_iterations": int(st.network_iterations),
               "network_off_at": int(st.network_off_at), "true_rel_residual": info.true_rel_residual,
               "us_per_iteration": 1e3 * statistics.mean(ms) / max(1, info.iterations),
               "training": {k: meta.get(k) for k in ("loads", "epochs", "steps", "batch", "lr", "val_loss_before",
                                                     "val_loss", "train_ms", "params", "held_out")}}
        x_main = x_dev.cpu().numpy().copy()
        # the same loop without the network
        for mode, name in ((_lib.LEARNED_SMOOTHING_ONLY, "without_network_smoothing_only"),
                           (_lib.LEARNED_BLOCK_JACOBI, "without_network_block_jacobi")):
            o2 = learned.solve_options(LEARNED_TOL, max_iterations=20000)
            i2, _ = ls.learned.solve_device(o2, F_dev.data_ptr(), x_dev.data_ptr(), mode)
            out[name] = {"iterations": int(i2.iterations), "ms": float(i2.solve_ms)}
        out["iteration_gain_vs_smoothing_only"] = (out["without_network_smoothing_only"]["iterations"] /
                                                   max(1, out["iterations"]))
        if chk is not None:
            errs = [float(np.linalg.norm(x_main - chk["truth"]) / np.linalg.norm(chk["truth"]))]
            if extra_F is not None:
                for f in extra_F:
                    ls.learned.solve_device(opts, f.data_ptr(), x_dev.data_ptr())
                    xt = chk["solve"](f.cpu().numpy())[0]
                    errs.append(float(np.linalg.norm(x_dev.cpu().numpy() - xt) / np.linalg.norm(xt)))
            out["accuracy"] = {"loads": {"count": len(errs), "rel_l2_max": max(errs),
                                         "rel_l2_p50": float(np.percentile(errs, 50)),
                                         "rel_l2_p99": float(np.percentile(errs, 99))}}
        # held-out loads: iterations and device time (errors against FP64
        # two-level solutions to 1e-12)
        k_h = min(args.learned_held_out, 512)
        if k_h > 0:
            H = learned_loads(wl, k_h)
            xt = learned.tight_solutions(torch, ctx, ls, H)
            rows = learned.evaluate(torch, ls, H, tolerance=LEARNED_TOL, truth=xt)
            its = [r["iterations"] for r in rows]
            out["held_out"] = {"loads": k_h, "seed": learned.HELD_OUT_SEED,
                               "iterations_p50": float(np.median(its)), "iterations_max": int(max(its)),
                               "ms_p50": float(np.median([r["ms"] for r in rows])),
                               "ms_p99": float(np.percentile([r["ms"] for r in rows], 99)),
                               "converged": int(sum(r["converged"] for r in rows)),
                               "rel_l2_max_vs_fp64_1e-12": max(r["rel_l2"] for r in rows),
                               "network_off": int(sum(r["network_off_at"] >= 0 for r in rows))}
        out["network_forward"] = network_forward_rate(ls.net, local)
    finally:
        ls.close()
    return out


def learned_loads(wl, k):
    from plategpu import learned, workloads

    return workloads.random_field_loads(wl, k, learned.HELD_OUT_SEED)


def network_forward_rate(net, local):
    """Device time of the network's forward pass (pg_net_forward, including
    the FP32 <-> BF16 packing) at batch 1 and 32, and the convolutions'
    FLOP rate at batch 32 against the measured BF16 peak."""
    import torch

    from plategpu import _lib

    from plategpu import learned

    H, W = net.height, net.width
    flops_px = learned.flops_per_image(H, W)
    res = {"flop_per_image": flops_px}
    for B in (1, 32):
        x = torch.randn(B, H, W, 3, device=f"cuda:{local}")
        y = torch.empty_like(x)
        for _ in range(3):
            net.forward(B, x.data_ptr(), y.data_ptr())
        torch.cuda.synchronize()
        s_, e_ = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        reps = 20
        s_.record()
        for _ in range(reps):
            net.forward(B, x.data_ptr(), y.data_ptr())
        e_.record()
        torch.cuda.synchronize()
        ms = s_.elapsed_time(e_) / reps
        res[f"batch{B}_us"] = 1e3 * ms
        res[f"batch{B}_tflops"] = flops_px * B / (ms * 1e-3) / 1e12
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            peak = float(json.load(f)["bf16_tflops"])
        res["bf16_peak_tflops"] = peak
        res["batch32_frac_of_bf16_peak"] = res["batch32_tflops"] / peak
    except (OSError, KeyError, ValueError):
        pass
    return res


def _lib_options_copy(o, **changes):
    """A copy of a PgOptions with some fields changed."""
    import ctypes

    c = type(o)()
    ctypes.memmove(ctypes.byref(c), ctypes.byref(o), ctypes.sizeof(o))
    for k, v in changes.items():
        setattr(c, k, v)
    return c


OTHER_VARIANTS = ("fp64", "mixed", "fp64_two_level", "mixed_two_level_cheb")


def other_configs_bench(args, ctx, stream, flush, world, local, check):
    """The other single-plate configs (plate_q4_32, plate_dkt_200, and the
    unstructured plate_holes_dkt), timed like
    the headline (device-resident solves, L2 flushed between steps, a quarter
    of the steps): plain FP64 block Jacobi (the reference's method) and three
    faster methods at the config's own stop tolerances; FP64-checked error of
    each when the checker runs; `best` is the fastest whose error is <= 1e-6
    (without the checker: whose true residual met its tolerance)."""
    import argparse

    import numpy as np
    import torch

    from plategpu import _lib, workloads

    out = {}
    for name in ("plate_q4_32", "plate_dkt_200", "plate_holes_dkt", "plate_q4_400"):
        if name == args.workload:
            continue
        wl = workloads.WORKLOADS[name]()
        sub = argparse.Namespace(**vars(args))
        sub.tol_bj, sub.tol_tl = TOLERANCES[name]
        sub.steps = max(3, args.steps // 4)
        prob = _lib.Problem(wl.mesh, wl.material, wl.coloring, wl.F, wl.cons_mask)
        F_dev = torch.from_numpy(wl.F).to(f"cuda:{local}")
        x_dev = torch.zeros(wl.n_dof, dtype=torch.float64, device=f"cuda:{local}")
        res, skipped = {}, {}
        for v in OTHER_VARIANTS:
            try:
                res[v] = time_variant(sub, world, local, ctx, prob, v, stream, F_dev, x_dev, flush)
            except _lib.PlateGPUError as e:  # e.g. a layout that does not fit this plate
                skipped[v] = str(e)
        chk = oracle_checks(wl, want_baseline=False) if check and name != "plate_q4_400" else None
        rows = {}
        for v, r in res.items():
            rows[v] = {k: r[k] for k in ("value", "kernel_ms", "iterations", "tolerance", "true_rel_residual",
                                         "global_path")}
            if r["global_path"]:
                # flexible PCG over global memory: 16 FP32 vector words per DOF and
                # iteration (the fewest vector reads and writes a PCG iteration
                # needs) against the HBM copy peak
                alg = 16.0 * 4 * wl.n_dof * max(1, r["iterations"])
                ach = alg / (r["kernel_ms"] * 1e-3) / 1e9
                rows[v]["roofline"] = {"achieved": ach, "peak": hbm_peak()[0], "unit": "GB/s",
                                       "frac": ach / hbm_peak()[0], "algorithmic_bytes": alg}
            if chk is not None:
                rows[v]["rel_l2_vs_fp64_truth"] = accuracy(r["x"], chk)["rel_l2_vs_fp64_truth"]

        def meets(v):
            e = rows[v].get("rel_l2_vs_fp64_truth")
            return e <= 1e-6 if e is not None else rows[v]["true_rel_residual"] <= rows[v]["tolerance"]

        if not rows:
            out[name] = {"unsupported": skipped}
            continue
        ok = [v for v in rows if meets(v)] or list(rows)
        best = min(ok, key=lambda v: rows[v]["value"])
        out[name] = {"dof": wl.n_dof, "elements": wl.mesh.elementCount,
                     "nodes_per_element": wl.mesh.nodesPerElement, "steps": sub.steps,
                     "best": best, "best_ms": rows[best]["value"], "variants": rows,
                     "skipped": skipped, "data": WORKLOAD_DATA.get(name)}
        del F_dev, x_dev
    return out


def case_loads(wl, k, seed=21):
    """k loads of the workload plate: its own load first, then seeded
    pressures with 16 point loads each (BCs applied)."""
    import numpy as np
    from plategpu import problem

    rng = np.random.default_rng(seed)
    out = [wl.F]
    for _ in range(k - 1):
        F = problem.pressure_load_vector(wl.mesh, rng.uniform(1e3, 8e3))
        for n in rng.choice(wl.mesh.nodeCount, 16, replace=False):
            F[3 * int(n)] += rng.uniform(1e3, 1e4)
        F32 = F.astype(np.float32)
        problem.applyBCsToRHS(F32, wl.constrainedDOFs)
        out.append(F32)
    return np.stack(out)


def cases_bench(args, ctx, wl, prob, H, method, check, world=1, local=0):
    """Load cases: args.cases loads of the workload plate through
    pg_solve_load_cases with the headline method (several cases in lockstep
    per persistent launch).  Device time of the launches and host wall clock
    of the whole call, per case, against the same loads solved one by one
    through pg_solve; FP64 error of every case when the checker runs."""
    import numpy as np

    F = case_loads(wl, args.cases)
    # the seeded loads need a tighter stop than the workload's own load for
    # an FP64-checked error of 1e-6 (5e-6 leaves up to 1.4e-6)
    opts = _lib_options_copy(H["opts"], tolerance=min(H["opts"].tolerance, 2e-6))
    for _ in range(2):
        ctx.solve_load_cases(prob, F, opts)
    dev, wall, one_dev, one_wall, last = [], [], [], [], None
    for _ in range(max(1, args.cases_steps)):
        barrier(world)
        t0 = time.perf_counter()
        X, infos = ctx.solve_load_cases(prob, F, opts)
        wall.append(max_over_ranks(world, (time.perf_counter() - t0) * 1e3, local))
        # the cases of one launch share its solve_ms
        launches = {}
        for i, inf in enumerate(infos):
            launches.setdefault((inf.solve_ms, inf.setup_ms), i)
        dev.append(max_over_ranks(world, sum(k[0] for k in launches), local))
        last = (X, infos)
        # the same loads one by one (pg_solve)
        barrier(world)
        t0 = time.perf_counter()
        d = 0.0
        for f in F:
            prob.set_F(f)
            d += ctx.solve(prob, opts)[1].solve_ms
        one_wall.append(max_over_ranks(world, (time.perf_counter() - t0) * 1e3, local))
        one_dev.append(max_over_ranks(world, d, local))
    prob.set_F(wl.F)
    X, infos = last
    k = args.cases
    out = {"cases": k, "method": method, "stop": f"||r||/||b|| < {opts.tolerance:g}",
           "device_ms_per_case": statistics.median(dev) / k,
           "e2e_ms_per_case": statistics.median(wall) / k,
           "one_by_one_device_ms_per_case": statistics.median(one_dev) / k,
           "one_by_one_e2e_ms_per_case": statistics.median(one_wall) / k,
           "iterations": [int(i.iterations) for i in infos],
           "reliable_updates": [int(i.reliable_updates) for i in infos],
           "fallbacks": int(sum(i.fallback for i in infos)),
           "shared_bytes": int(infos[0].shared_bytes),
           "h2d_bytes": int(F.nbytes), "d2h_bytes": int(8 * F.size)}
    out["speedup_device"] = out["one_by_one_device_ms_per_case"] / out["device_ms_per_case"]
    out["speedup_e2e"] = out["one_by_one_e2e_ms_per_case"] / out["e2e_ms_per_case"]
    if check:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O
        m, mat = wl.mesh, wl.material
        ke = O.all_ke(m.nodes, m.elements, m.nodesPerElement, mat.E, mat.nu, mat.t, elem_t=mat.elem_t,
                      mode=O.FP64)
        errs = []
        for f, x in zip(F, X):
            xt, _ = O.truth_solve(m.nodeCount, m.elements, m.nodesPerElement, ke, wl.cons_mask,
                                  f.astype(np.float64))
            errs.append(float(np.linalg.norm(x - xt) / np.linalg.norm(xt)))
        out["rel_l2_vs_fp64_truth"] = errs
    return out


BATCH_METHODS = ("mixed_two_level", "fp64_two_level", "fp64_two_level_cheb", "fp64_block_jacobi")


def batch_options(name, part_nodes=0):
    """Options of one batch method: the stop is ||r||/||b|| < 2e-7 for all
    (the DKT plates need a tighter residual than the Q4 ones for 1e-6 error);
    part_nodes: the team-size target (0 = the library's default)."""
    from plategpu import _lib

    prec = _lib.PG_PREC_MIXED if name.startswith("mixed") else _lib.PG_PREC_FP64
    pre = _lib.PG_PRECOND_BLOCK_JACOBI if name.endswith("block_jacobi") else _lib.PG_PRECOND_TWO_LEVEL
    smo = _lib.PG_SMOOTHER_CHEBYSHEV if name.endswith("cheb") else _lib.PG_SMOOTHER_BLOCK_JACOBI
    return _lib.make_options(tolerance=2e-7, max_iterations=50000, stop_rule=_lib.PG_STOP_RELATIVE,
                             precision=prec, preconditioner=pre, smoother=smo, batch_part_nodes=part_nodes)


def batch_bench(args, ctx, check, world=1, rank=0, local=0):
    """The uneven-plate batch (batched solver, one persistent launch per
    phase), timed for several methods: mixed-precision two-level (plates
    whose mixed solve stagnates finish with an FP64 correction), FP64
    two-level with and without the Chebyshev smoother, and the reference's
    FP64 block Jacobi (one timed solve).  For each: solves/s, per-plate p50 /
    p99 / max, and the FP64 error on a seeded sample of plates when the
    checker runs.  The headline is the fastest method whose sampled errors
    are <= 1e-6.  With N ranks the plates are shared out by estimated cost
    (no collective on the data path); the batch time is the largest over the
    ranks, and every rank takes the same collective steps."""
    import numpy as np
    from plategpu import _lib, workloads

    ALL = workloads.batch_uneven(count=args.batch)
    shards = workloads.shard_lpt([workloads.plate_cost(w) for w in ALL], world)
    B = [ALL[i] for i in shards[rank]]
    probs = [_lib.Problem(w.mesh, w.material, w.coloring, w.F, w.cons_mask) for w in B]
    truth_jobs, pool = {}, None
    if check:
        # FP64 truth (sparse LU) of a sample: the 5 largest plates and a
        # seeded 5% of the others, computed by worker processes while the GPU
        # runs
        import concurrent.futures as cf
        import multiprocessing as mp
        rng = np.random.default_rng(11)
        by_size = sorted(range(len(B)), key=lambda i: -B[i].mesh.nodeCount)
        rest = by_size[5:]
        pick = by_size[:5] + rng.choice(rest, size=min(len(rest), max(6, (len(B) + 19) // 20)),
                                        replace=False).tolist()
        pool = cf.ProcessPoolExecutor(max_workers=min(len(pick), max(1, (os.cpu_count() or 2) - 1), 16),
                                      mp_context=mp.get_context("spawn"))
        for i in pick:
            w = B[i]
            m, mat = w.mesh, w.material
            truth_jobs[i] = pool.submit(_truth_job, m.nodeCount, m.nodes, m.elements, m.nodesPerElement,
                                        mat.E, mat.nu, mat.t, mat.elem_t, w.cons_mask, w.F)
    methods = BATCH_METHODS if args.batch_fp64 else BATCH_METHODS[:1]
    rows, per_plate, fallback_plates, truth_note = {}, {}, [], None
    # the team-size target, tuned on this GPU for this batch (FP64 two-level)
    # by plategpu.autotune and cached per GPU name and batch
    import torch
    from plategpu import autotune
    part_nodes, tune = autotune.tune_batch(
        ctx, probs, batch_options("fp64_two_level"), torch.cuda.get_device_name(local),
        candidates=(100, 160, 200, 400), cache_path=os.path.join(tempfile.gettempdir(), "plategpu_autotune.json"))
    for name in methods:
        opts = batch_options(name, part_nodes)
        steps = 1 if name == "fp64_block_jacobi" else max(1, args.batch_steps)
        ms, last, err = [], None, None
        try:  # every rank reaches the collectives below whatever happens here
            b = ctx.batch(probs, opts)
            b.solve(opts, want_x=False)  # first solve: coarse matrices, set-up kernels
            for k in range(steps):
                last = b.solve(opts, want_x=(k == steps - 1))
                ms.append(last[2].solve_ms)
            b.close()
        except _lib.PlateGPUError as e:
            err = str(e)
        failed = max_over_ranks(world, 1.0 if err else 0.0, local)
        t = [max_over_ranks(world, 0.0 if err else ms[k], local) for k in range(steps)]
        if failed:
            rows[name] = {"unavailable": err or "failed on another rank"}
            continue
        xs, infos, bi = last
        if check and name == methods[0]:
            # plates that stagnated in mixed precision and were finished by
            # the FP64 correction
            fallback_plates = [i for i, inf in enumerate(infos) if inf.fallback]
        med = statistics.median(t)
        its = [i.iterations for i in infos]
        row = {"solves_per_s": len(ALL) / (med * 1e-3), "batch_ms": med, "batch_ms_all": t,
               "plate_ms_p50": bi.plate_ms_p50, "plate_ms_p99": bi.plate_ms_p99,
               "plate_ms_max": bi.plate_ms_max, "phases": bi.phases, "teams": bi.teams,
               "cuda_graph": int(bi.graph),
               "fallbacks_rank0": bi.fallbacks, "converged_rank0": bi.converged,
               "iterations_median": float(np.median(its)), "iterations_max": int(max(its))}
        if check:
            per_plate[name] = xs
        rows[name] = row

    if check:
        # every plate of every method against an FP64 two-level solve of the
        # same plate to ||r||/||b|| < 1e-12 (the LU truths below pin that
        # solve), and the LU-truth sample
        tight = batch_options("fp64_two_level")
        tight.tolerance = 1e-12
        tb = ctx.batch(probs, tight)
        xt_all = tb.solve(tight)[0]
        tb.close()
        truths = {i: f.result()[0] for i, f in truth_jobs.items()}
        pool.shutdown()
        for name, xs in per_plate.items():
            errs = [float(np.linalg.norm(x - t) / np.linalg.norm(t)) for x, t in zip(xs, xt_all)]
            rows[name]["rel_l2_vs_fp64_tight_all"] = {
                "plates": len(errs), "max": max(errs), "p50": float(np.median(errs)),
                "worst_plate": B[int(np.argmax(errs))].name}
            samp = {B[i].name: float(np.linalg.norm(xs[i] - t) / np.linalg.norm(t))
                    for i, t in truths.items()}
            rows[name]["rel_l2_vs_fp64_truth_sample"] = samp
            rows[name]["max_rel_l2_vs_fp64_truth"] = max(samp.values())
            if name == methods[0]:
                fb = [float(np.linalg.norm(xs[i] - xt_all[i]) / np.linalg.norm(xt_all[i]))
                      for i in fallback_plates]
                rows[name]["fallback_plates_rel_l2_vs_fp64_tight_max"] = max(fb) if fb else None
        tight_vs_truth = [float(np.linalg.norm(xt_all[i] - t) / np.linalg.norm(t)) for i, t in truths.items()]
        truth_note = {"sample_plates": len(truths),
                      "sample": "the 5 largest plates and a seeded 5% of the others (sparse LU)",
                      "tight_fp64_vs_truth_max": max(tight_vs_truth) if tight_vs_truth else None}

    def meets(name):
        r = rows[name]
        if "unavailable" in r or r["converged_rank0"] != len(B):
            return False
        e = r.get("rel_l2_vs_fp64_truth_sample")
        a = r.get("rel_l2_vs_fp64_tight_all")
        return (e is None or max(e.values()) <= 1e-6) and (a is None or a["max"] <= 1e-6)

    ok = [n for n in rows if meets(n)] or [n for n in rows if "unavailable" not in rows[n]]
    head = min(ok, key=lambda n: rows[n]["batch_ms"])
    out = {"workload": ("batch_uneven: %d plates, elements per side log-uniform 16-256, 70%% Q4 / "
                        "30%% DKT, random material, supports and random-field loads" % len(ALL)),
           "dof_total": int(sum(3 * w.mesh.nodeCount for w in ALL)),
           "ranks": world, "plates_per_rank": [len(sh) for sh in shards],
           "method": head, "stop": "||r||/||b|| < 2e-7",
           "autotune": {"batch_part_nodes": part_nodes, "times_ms": tune["times_ms"],
                        "cached": tune["cached"]}}
    out.update(rows[head])
    out["methods"] = rows
    if check:
        out["accuracy_check"] = truth_note
    return out


def _truth_job(Nn, nodes, elements, npe, E, nu, t, elem_t, cons, F):
    """FP64 truth of one plate (oracle, in a worker process)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O

    ke = O.all_ke(nodes, elements, npe, E, nu, t, elem_t=elem_t, mode=O.FP64)
    return O.truth_solve(Nn, elements, npe, ke, cons, F)


def main():
    args = parse_args()
    world, rank, local = dist_setup(args)
    try:
        if args.impl == "reference":
            run_reference(args, world, rank)
        else:
            run_plategpu(args, world, rank, local)
    finally:
        if world > 1:
            import torch.distributed as dist

            dist.destroy_process_group()


if __name__ == "__main__":
    main()
