"""Benchmark of the plain FP64 MHD step (HLLD, minmod, Heun RK2) on a 256^3 Cartesian grid.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--n 256]
                    [--tsteps 200]

One bench step = one solve of the workload: restart from the resident seeded initial state
(a 1.07 GB device-to-device copy) and run `--tsteps` (200) time steps of the 256^3 grid.
Prints one JSON line on rank 0.

  value     cell-updates/s over the K timed solves, state resident in HBM (1.07 GB per buffer,
            far above the 126 MB L2), CUDA events on the solver's stream, max over ranks.
  e2e       the same metric through the C ABI with host buffers: every step uploads Cell_par
            (setb_set_state, pinned host memory), runs the solve, downloads Cell_par
            (setb_get_state); device-timed with events on the solver's stream.
  roofline  per-kernel CUDA-event times over the timed region (setb_step_profiled); algorithmic
            bytes per cell-update: 128 B for the first stage (read U^n, write U*), 192 B for the
            second (read U*, U^n, write U^n+1).
  c3        config C3: one seeded Mach/beta draw at 384^3 x 500 steps, the mixed form against
            plain FP64 (speed-up, L1 of rho, p, |B|, total-energy drift).
  cpu_baseline  the CPU oracle (a port of the reference algorithm) on this host's cores: one
            RK2 step of the same grid, plus the 96^3 parity grid and config C1 (64^3, first
            order, forward Euler) at all threads and one thread.
`--c5 K` runs config C5 at its stated parameters on K requests instead (one JSON line).
N > 1 runs N independent replicas (weak scaling): no data-path collective.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

BYTES_STAGE1 = 128   # read U^n (8 x f64), write U* (8 x f64)
BYTES_STAGE2 = 192   # read U*, U^n, write U^n+1
BYTES_STEP = BYTES_STAGE1 + BYTES_STAGE2
# DRAM bytes (read + write) per cell of one plain stage-2 launch, from an ncu capture of that
# kernel at 160^3 (dram__bytes_read.sum 546.3 MB + dram__bytes_write.sum 225.9 MB over 4.096 M
# cells); traffic grows with the cell count, so the full-size launch's traffic is this figure
# times its cells.
TRAFFIC_STAGE2_PER_CELL = 772.2e6 / 160 ** 3
# FP64 pipe thread instructions (DFMA + DMUL + DADD + DSETP) per cell of the same launch, from
# the same capture's opcode counts (107.18 M warp instructions x 31.87 threads / 4.096 M cells).
FP64_OPS_STAGE2_PER_CELL = 834


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clock / throttle sampling during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.path = None

    def __enter__(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200", "-f", self.path], stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.path or not os.path.exists(self.path):
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        sm, smax, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = float(parts[2])
            except ValueError:
                continue
            for nm, val in zip(names, parts[5:9]):
                if val.lower() == "active":
                    reasons.add(nm)
        os.unlink(self.path)
        busy = [x for x in sm if smax and x > 0.3 * smax] or sm
        return {"sm_mhz": statistics.median(busy) if busy else None, "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_setup():
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return world, rank, local


def cpu_baseline(n: int, tsteps_sample: int = 1, threads: int = 0, order: int = 2, scheme: int = 2,
                 seed: int = 2, developed: bool = True):
    """The oracle (CPU port of the reference algorithm) on `threads` host threads (0 = all):
    `tsteps_sample` HLLD steps (minmod + Heun RK2 by default, or first order + forward Euler) of
    the n^3 grid; returns cell-updates/s, the thread count and the seconds.  `developed` starts
    from dt = 1e-4 instead of the reference's 2e-9 first step (the rate does not depend on dt)."""
    import oracle as O
    O.build()
    g = O.make_grid(n, r_floor=0.5 * 2.0 / n)
    U = O.init_lism(g, seed=seed)
    ck = O.clock_init(g)
    if developed:
        ck.dt_next = 1e-4
    threads = threads or O.max_threads()
    t0 = time.perf_counter()
    O.run(g, O.make_opts(3, order, scheme, 0.4), U, tsteps_sample, ck, nthreads=threads)
    dt = time.perf_counter() - t0
    return n ** 3 * tsteps_sample / dt, threads, dt


def cpu_baseline_line(n: int):
    """The CPU baselines: the bench workload's grid (one RK2 step, all threads) as `value`, the
    C2 parity grid (96^3, RK2) and config C1 (64^3, first order, forward Euler, 100 steps) at all
    threads and one thread (bounded samples, ~15-25 s of CPU work in all)."""
    v, thr, secs = cpu_baseline(n)
    c2a, _, s2a = cpu_baseline(96, tsteps_sample=10)
    c2b, _, s2b = cpu_baseline(96, tsteps_sample=1, threads=1)
    c1a, _, s1a = cpu_baseline(64, tsteps_sample=100, order=1, scheme=1, seed=1, developed=False)
    c1b, _, s1b = cpu_baseline(64, tsteps_sample=10, order=1, scheme=1, seed=1, developed=False, threads=1)
    return {"value": v, "unit": "cell-updates/s", "cores": thr, "kind": "port",
            "sample": f"1 RK2 HLLD minmod step of the {n}^3 grid ({secs:.1f} s)",
            "c2_96": {"all_threads": c2a, "cores": thr, "one_thread": c2b, "unit": "cell-updates/s",
                      "sample": f"96^3 RK2 HLLD minmod: 10 steps on all threads ({s2a:.1f} s), 1 step on one "
                                f"thread ({s2b:.1f} s)"},
            "c1": {"all_threads": c1a, "cores": thr, "one_thread": c1b, "unit": "cell-updates/s",
                   "sample": f"C1 64^3 first-order HLLD forward Euler: 100 steps on all threads ({s1a:.1f} s), "
                             f"10 steps on one thread ({s1b:.1f} s)"}}


def run_reference(args, world, rank):
    """`--impl reference`: the reference algorithm's CPU implementation (the oracle port; the
    CUDA Fortran reference needs nvfortran, which this image lacks) on this host's cores."""
    if rank != 0:
        return
    import oracle as O
    O.build()
    n = args.n
    g = O.make_grid(n, r_floor=0.5 * 2.0 / n)
    U = O.init_lism(g, seed=2)
    ck = O.clock_init(g)
    ck.dt_next = 1e-4
    threads = O.max_threads()
    o = O.make_opts(3, 2, 2, 0.4)
    for _ in range(args.warmup):
        O.run(g, o, U, 1, ck, nthreads=threads)
    t0 = time.perf_counter()
    for _ in range(args.steps):
        O.run(g, o, U, 1, ck, nthreads=threads)
    dt = time.perf_counter() - t0
    value = n ** 3 * args.steps / dt
    line = {
        "metric": "cell_updates_per_s", "value": value, "unit": "cell-updates/s", "impl": "reference",
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * dt / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": config_dict(args, reference=True),
        "cpu_baseline": {"value": value, "unit": "cell-updates/s", "cores": threads, "kind": "port",
                         "sample": f"1 RK2 HLLD minmod step of the {n}^3 grid per bench step, dt 1e-4 (the "
                                   f"GPU arm's bench step is a {args.tsteps}-step solve; the metric is a rate)"},
        "e2e": {"value": value, "unit": "cell-updates/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def config_dict(args, reference=False):
    tps = 1 if reference else args.tsteps
    return {"workload": f"C2 plain FP64: ideal MHD, HLLD + minmod + Heun RK2, {args.n}^3 Cartesian, "
                        f"{tps} time step{'s' if tps > 1 else ''} per bench step",
            "grid": [args.n] * 3, "time_steps_per_step": tps, "n_state": 3, "order": 2, "scheme": "rk2",
            "cfl": 0.4, "precision": "plain-fp64",
            "l2": "inputs larger than L2 (state 1.07 GB per buffer at 256^3)",
            "parallelism": f"replicas{args.gpus}" if args.gpus > 1 else "single"}


def facelist_leg(n: int, tsteps: int, permute: bool):
    """The face-list path (the reference's own geometry) on an n^3 box of the C2 physics, cells and
    faces in natural order or renumbered at random: cell-updates/s from CUDA events around every
    stage (3 launches each), and the DRAM bytes per cell-update a stage needs at least."""
    from set_b200 import facelist as FL
    m = FL.box_facelist((n, n, n), seed=1, permute_seed=7 if permute else None,
                        sides={"x-": 4, "x+": 4, "y-": 4, "y+": 4, "z-": 4, "z+": 4})
    params = FL.fl_params(r_src=0.125, rho_src=50.0, v_src=10.0, p_over_rho_src=0.01, r_floor=1.0 / n, dt_init=2e-9)
    cp = FL.lism_cellpar(m, seed=2, params=params)
    o = __import__("set_b200").step_opts(n_state=3, order=2, scheme=2, cfl=0.4)
    with FL.FaceListSolver(m, cp, params) as s:
        s.step(5, o)
        _, ms, cnt = s.step_profiled(tsteps, o)
        diag = s.status()
    cells = m.n_cell
    return {"grid": f"{n}^3 box, {'random' if permute else 'natural'} numbering", "cells": cells,
            "faces": m.n_gran, "time_steps": tsteps, "cell_updates_per_s": cells * tsteps / (sum(ms) / 1e3),
            "stage1_ms": ms[0] / max(cnt[0], 1), "stage2_ms": ms[1] / max(cnt[1], 1),
            "n_negdens": diag.n_negdens}


def run_mixed_only(args):
    """`--mixed-only`: only the mixed-form leg (W warm-up and K timed solves); used to profile the
    mixed kernel in isolation."""
    import set_b200 as S
    n, T = args.n, args.tsteps
    desc = S.cart_desc(n)
    ic = S.lism_ic(seed=2)
    o = S.step_opts(n_state=3, order=2, scheme=2, cfl=0.4, precision=args.mixed_precision)
    with S.Solver(desc, ic=ic) as s, S.Solver(desc, ic=ic) as ic_state:
        for _ in range(args.warmup):
            s.copy_from(ic_state)
            s.step(T, o)
        ms = [0.0, 0.0]
        cnt = [0, 0]
        for _ in range(args.steps):
            s.copy_from(ic_state)
            _, m, c = s.step_profiled(T, o)
            ms = [ms[i] + m[i] for i in range(2)]
            cnt = [cnt[i] + c[i] for i in range(2)]
    print(json.dumps({"leg": f"mixed{args.mixed_precision}", "grid": n, "stage1_ms": ms[0] / max(cnt[0], 1),
                      "stage2_ms": ms[1] / max(cnt[1], 1),
                      "cell_updates_per_s": n ** 3 * T * args.steps / (sum(ms) / 1e3)}), flush=True)


def run_c5(args):
    """`--c5 K`: config C5 at its stated parameters on the first K requests of the seeded stream
    (Poisson 20/s, cubic edges log-uniform [32,256], 30 % hydro / 70 % MHD, steady state when the
    relative L1 change of rho between 50-step checks is below 1e-5, cap 3000 steps, CFL 0.2, 150 GB
    admission budget), served in the mixed form by the native continuous-batching server, then the
    same requests solved one at a time in the plain FP64 form.  Reports latency percentiles,
    solves/s, convergence and failures, and the served-vs-plain L1 of rho for every request that
    both ran to the same step count (states kept for edges <= 160 to bound host memory)."""
    import numpy as np
    import set_b200  # noqa: F401  (fails loudly without the CUDA library)
    from set_b200 import workloads as WL, serve as SV
    reqs = WL.c5_requests(count=args.c5, rate=20.0, lo=32, hi=256, max_steps=3000)
    keep = [k for k, r in enumerate(reqs) if r.inst.desc.nx <= 160]
    out = SV.run_stream(reqs, max_slots=256, precision=1, keep=keep)
    SV.warm_kernels(reqs, 0)   # the plain kernels' first-use loading stays out of the timed loop
    t0 = time.perf_counter()
    l1, same_steps, seq_steps, seq_conv, seq_failed, both_failed = [], 0, [], 0, 0, 0
    for k, rq in enumerate(reqs):
        alone = SV.solve_alone(rq.inst, 0, rq.steady_tol, rq.max_steps, keep_state=k in out["states"])
        seq_steps.append(alone["steps"])
        seq_conv += int(alone["converged"])
        seq_failed += int(alone["status"] != 0)
        both_failed += int(alone["status"] != 0 and out["results"][k].status != 0)
        if (k in out["states"] and alone["steps"] == out["steps"][k] and out["results"][k].status == 0
                and alone["status"] == 0):
            a, b = alone["U"][0], out["states"][k][0]
            l1.append(float(np.abs(b - a).sum() / np.abs(a).sum()))
            same_steps += 1
    seq_secs = time.perf_counter() - t0
    edges = [r.inst.desc.nx for r in reqs]
    line = {"leg": "C5", "config": {"requests": len(reqs), "rate_per_s": 20.0, "edges": "cubic, log-uniform [32,256]",
                                    "hydro_fraction": 0.3, "steady_tol": 1e-5, "check_every": 50, "max_steps": 3000,
                                    "cfl": 0.2, "hbm_budget_bytes": 150 * 10 ** 9, "served_precision": "mixed",
                                    "edge_min_max": [min(edges), max(edges)]},
            "latency_p50_s": out["latency_p50_s"], "latency_p99_s": out["latency_p99_s"],
            "solves_per_s": out["solves_per_s"], "span_s": out["span_s"], "max_active": out["max_active"],
            "converged": out["converged"], "failed": out["failed"], "failed_by_status": out["failed_by_status"],
            "steps_mean": float(np.mean(out["steps"])),
            "sequential_plain_solves_per_s": len(reqs) / seq_secs, "sequential_plain_seconds": seq_secs,
            "sequential_plain_converged": seq_conv, "sequential_plain_failed": seq_failed,
            "failed_in_both": both_failed,
            "speedup_vs_sequential_plain": out["solves_per_s"] / (len(reqs) / seq_secs),
            "l1_rho_served_vs_plain": {"compared": same_steps, "max": max(l1) if l1 else None,
                                       "median": float(np.median(l1)) if l1 else None}}
    print(json.dumps(line), flush=True)


def run_slab(args, world, rank, local):
    """One grid of n x n x (n * ranks) cells split along z, one n^3 slab per rank, ghost planes
    exchanged over NCCL each stage and the dt minimum all-reduced each step (weak scaling)."""
    import numpy as np
    import torch
    import set_b200 as S
    from set_b200 import slab as SL

    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        torch.distributed.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
        torch.distributed.barrier()   # a group-wide collective before the first point-to-point batch
    n, T = args.n, args.tsteps
    nz = n * world
    desc = S.cart_desc((n, n, nz))
    k0, nl = SL.split_z(nz, world)[rank]
    rng = np.random.default_rng(2 + rank)   # this rank's planes only (the whole grid needs not fit a host)
    cp = np.zeros((n * n * nl, 16))
    cp[:, :8] = S.lism_prim()
    cp[:, 0] *= 1.0 + 1e-3 * rng.uniform(-1.0, 1.0, n * n * nl)
    cp[:, 4] *= 1.0 + 1e-3 * rng.uniform(-1.0, 1.0, n * n * nl)
    slab, ic = SL.SlabSolver(desc, k0, nl, cp), SL.SlabSolver(desc, k0, nl, cp)
    run = SL.SlabRun(slab, rank, world)
    opts = S.step_opts(n_state=3, order=2, scheme=2, cfl=0.4)
    stream = torch.cuda.ExternalStream(slab.stream())

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    for _ in range(args.warmup):
        slab.copy_from(ic)
        run.step(T, opts)
    barrier()
    torch.cuda.synchronize()
    with ClockSampler(local) as clk:
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(args.steps):
            slab.copy_from(ic)
            run.step(T, opts)
        ev1.record(stream)
        ev1.synchronize()
    torch.cuda.synchronize()
    barrier()
    ms = ev0.elapsed_time(ev1)
    if world > 1:
        t = torch.tensor([ms], dtype=torch.float64, device="cuda")
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        ms = float(t.item())
    diag = slab.status()
    cells = n * n * nz
    if rank == 0:
        line = {"metric": "cell_updates_per_s", "value": cells * T * args.steps / (ms / 1e3),
                "unit": "cell-updates/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": ms / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f64", "data": "synthetic (LISM + solar-wind source, seeded)",
                "config": {"workload": f"one grid split along z: {n}x{n}x{nz}, {n}^3 per GPU, HLLD + minmod + "
                                       f"Heun RK2, {T} time steps per bench step",
                           "grid": [n, n, nz], "time_steps_per_step": T, "parallelism": f"slab{world}",
                           "exchange": "2 ghost planes x 8 variables per neighbour and stage, dt min per step"},
                "clocks": clk.summary(), "gpu_launches": 2 * T * args.steps,
                "diag": {"time_all": diag.time_all, "n_negdens": diag.n_negdens}}
        print(json.dumps(line), flush=True)
    slab.close()
    ic.close()
    if world > 1:
        torch.distributed.destroy_process_group()


def run_ours(args, world, rank, local):
    import numpy as np
    import torch
    import set_b200 as S

    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        torch.distributed.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    n, T = args.n, args.tsteps
    desc = S.cart_desc(n)
    ic = S.lism_ic(seed=2 + rank)
    opts = S.step_opts(n_state=3, order=2, scheme=2, cfl=0.4)
    solver = S.Solver(desc, ic=ic)
    ic_state = S.Solver(desc, ic=ic)   # resident initial state each solve restarts from
    stream = torch.cuda.ExternalStream(solver.stream())
    cells = n ** 3

    def barrier():
        if world > 1:
            torch.distributed.barrier()

    def max_over_ranks(x):
        if world == 1:
            return x
        t = torch.tensor([x], dtype=torch.float64, device="cuda")
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
        return float(t.item())

    # ---- warm-up
    for _ in range(args.warmup):
        solver.copy_from(ic_state)
        solver.step(T, opts)

    # ---- device-resident timed region (per-kernel events inside setb_step_profiled)
    barrier()
    torch.cuda.synchronize()
    k_ms = [0.0, 0.0]
    k_n = [0, 0]
    with ClockSampler(local) as clk:
        ev0 = torch.cuda.Event(enable_timing=True)
        ev1 = torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(args.steps):
            solver.copy_from(ic_state)
            _, ms, cnt = solver.step_profiled(T, opts)
            k_ms = [k_ms[i] + ms[i] for i in range(2)]
            k_n = [k_n[i] + cnt[i] for i in range(2)]
        ev1.record(stream)
        ev1.synchronize()
    torch.cuda.synchronize()
    barrier()
    ms_total = max_over_ranks(ev0.elapsed_time(ev1))
    clocks = clk.summary()
    diag = solver.status()
    value = world * cells * T * args.steps / (ms_total / 1e3)

    hbm, peak_kind = peaks()
    t1 = k_ms[0] / max(k_n[0], 1)
    t2 = k_ms[1] / max(k_n[1], 1)
    ach2 = BYTES_STAGE2 * cells / (t2 / 1e3) / 1e9
    ach_step = BYTES_STEP * cells / ((t1 + t2) / 1e3) / 1e9
    # the pipe that bounds the kernel: FP64 operations of the stage-2 launch (counted by ncu)
    # against 64 FP64 lanes per SM per clock at the sampled SM clock
    sms = torch.cuda.get_device_properties(local).multi_processor_count
    sm_hz = (clocks.get("sm_mhz") or 1965.0) * 1e6
    fp64_ach = FP64_OPS_STAGE2_PER_CELL * cells / (t2 / 1e3) / 1e12
    fp64_peak = 64 * sms * sm_hz / 1e12

    # ---- mixed form on the same workload: speed and L1 density error against the plain run
    mixed = None
    if not args.no_mixed:
        def rho_after(prec, nsteps):
            with S.Solver(desc, ic=ic) as s2:
                s2.step(nsteps, S.step_opts(n_state=3, order=2, scheme=2, cfl=0.4, precision=prec))
                return s2.conserved()[0]
        solver_m = S.Solver(desc, ic=ic)
        opts_m = S.step_opts(n_state=3, order=2, scheme=2, cfl=0.4, precision=1)
        for _ in range(args.warmup):
            solver_m.copy_from(ic_state)
            solver_m.step(T, opts_m)
        barrier()
        torch.cuda.synchronize()
        mk = [0.0, 0.0]
        mn = [0, 0]
        for _ in range(args.steps):
            solver_m.copy_from(ic_state)
            _, ms, cnt = solver_m.step_profiled(T, opts_m)
            mk = [mk[i] + ms[i] for i in range(2)]
            mn = [mn[i] + cnt[i] for i in range(2)]
        mixed_ms = max_over_ranks(sum(mk))
        redo = solver_m.status().n_fp64_redo
        solver_m.close()
        r64 = rho_after(0, T)
        r32 = rho_after(1, T)
        l1 = float(np.abs(r32 - r64).sum() / np.abs(r64).sum())
        mixed = {"value": world * cells * T * args.steps / (mixed_ms / 1e3), "unit": "cell-updates/s",
                 "speedup_vs_plain": (sum(k_ms)) / sum(mk), "stage1_ms": mk[0] / max(mn[0], 1),
                 "stage2_ms": mk[1] / max(mn[1], 1), "l1_rho_vs_plain_fp64": l1, "l1_after_steps": T,
                 "fp64_face_recomputes": redo,
                 "hbm_gbs": 384 * cells / ((mk[0] + mk[1]) / max(mn[0], 1) / 1e3) / 1e9,
                 "algorithmic_bytes_per_cell_step": 384}

    # ---- end to end through the C ABI with host buffers
    cp = torch.empty((cells, 16), dtype=torch.float64, pin_memory=True).numpy()
    cp[:] = 0.0
    cp_init = S.fill_lism(desc, ic)
    cp[:, :] = cp_init
    for _ in range(1):
        solver.set_state(cp, 0.0)
        solver.step(T, opts)
        solver.get_state(cp)
    barrier()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        solver.set_state(cp, 0.0)
        solver.step(T, opts, wait=False)
        solver.get_state(cp)
    e1.record(stream)
    e1.synchronize()
    barrier()
    e2e_ms = max_over_ranks(e0.elapsed_time(e1))
    e2e = world * cells * T * args.steps / (e2e_ms / 1e3)
    finite = bool(np.isfinite(cp[:, :8]).all())

    # ---- config C4: the 64-grid ensemble (mixed, one batch) vs sequential plain-form solves
    ensemble = None
    if rank == 0 and world == 1 and not args.no_ensemble:
        from set_b200 import workloads as WL
        inst = WL.c4_instances()
        small = sorted(range(len(inst)), key=lambda k: inst[k].cells)[:4]
        bat = WL.run_batched(inst, tune=True, keep=small)
        seq = WL.run_sequential(inst, precision=0, keep=small)
        l1 = max(float(np.abs(bat["states"][k][0] - seq["states"][k][0]).sum() / np.abs(seq["states"][k][0]).sum())
                 for k in small)
        ensemble = {"config": "C4: 64 grids, edges log-uniform [48,160] per axis, HLLD RK2 minmod mixed, "
                              "300 steps, CFL 0.2",
                    "solves_per_s": bat["solves_per_s"], "seconds": bat["seconds"],
                    "cell_updates_per_s": bat["cell_updates_per_s"], "tuned": bat["tuned"],
                    "sequential_plain_solves_per_s": seq["solves_per_s"], "sequential_plain_seconds": seq["seconds"],
                    "speedup_vs_sequential_plain": bat["solves_per_s"] / seq["solves_per_s"],
                    "l1_rho_vs_plain_max_of_4_smallest": l1, "total_cells": sum(i.cells for i in inst),
                    "fp64_face_recomputes": bat["fp64_redo"], "n_negdens": bat["n_negdens"],
                    "n_negdens_sequential": seq["n_negdens"]}

    # ---- config C5 (scaled): a Poisson request stream through the solve server
    served = None
    if rank == 0 and world == 1 and args.serve_requests > 0:
        from set_b200 import workloads as WL, serve as SV
        reqs = WL.c5_requests(count=args.serve_requests, rate=20.0, lo=32, hi=args.serve_max_edge,
                              max_steps=args.serve_max_steps)
        out = SV.run_stream(reqs, max_slots=256, precision=1)
        seq = SV.run_sequential(reqs, precision=0)
        served = {"config": f"C5 scaled: {len(reqs)} requests, Poisson 20/s, cubic edge log-uniform "
                            f"[32,{args.serve_max_edge}], 30% hydro (HLLC) / 70% MHD (HLLD), steady state 1e-5 "
                            f"per 50-step check or cap {args.serve_max_steps} steps, CFL 0.2, 150 GB budget",
                  "latency_p50_s": out["latency_p50_s"], "latency_p99_s": out["latency_p99_s"],
                  "solves_per_s": out["solves_per_s"], "span_s": out["span_s"], "max_active": out["max_active"],
                  "converged": out["converged"], "failed": out["failed"],
                  "failed_by_status": out["failed_by_status"],
                  "sequential_plain_solves_per_s": seq["solves_per_s"],
                  "speedup_vs_sequential_plain": out["solves_per_s"] / seq["solves_per_s"]}

    # ---- the face-list path (the reference's own grid geometry) on a 128^3 box
    facelist = None
    if rank == 0 and world == 1 and args.facelist_n > 0:
        facelist = [facelist_leg(args.facelist_n, 50, False), facelist_leg(args.facelist_n, 50, True)]

    # ---- config C3: one seeded Mach / beta draw at 384^3 x 500 steps, mixed against plain FP64
    c3 = None
    if rank == 0 and world == 1 and args.c3_n > 0:
        from set_b200 import workloads as WL
        r = WL.run_c3(WL.c3_problems(count=1, n=args.c3_n, steps=args.c3_steps), mixed=(1,))[0]
        c3 = {"config": f"C3: {args.c3_n}^3, {args.c3_steps} steps, HLLD minmod Heun RK2, CFL 0.4, one seeded "
                        f"draw of LISM Mach in [2,8] and beta in [0.1,10] ({r['label']})",
              "plain_cell_updates_per_s": r["plain_cell_updates_per_s"], "mixed": r["mixed1"],
              "plain_n_negdens": r["plain_n_negdens"]}

    base = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        base = cpu_baseline_line(n)

    if rank == 0:
        line = {
            "metric": "cell_updates_per_s", "value": value, "unit": "cell-updates/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_total / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic: seeded LISM inflow + solar-wind source sphere (the reference measures no dataset)",
            "config": config_dict(args),
            "e2e": {"value": e2e, "unit": "cell-updates/s", "h2d_bytes_per_step": cells * 64,
                    "d2h_bytes_per_step": cells * 64},
            "roofline": {"bound": "hbm", "kernel": "stage_kernel<plain FP64, HLLD, minmod, Heun stage 2>",
                         "achieved": ach2, "peak": hbm, "unit": "GB/s", "frac": ach2 / hbm,
                         "peak_kind": peak_kind, "traffic": TRAFFIC_STAGE2_PER_CELL * cells,
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum at 160^3, "
                                           "scaled by cells",
                         "stage1_ms": t1, "stage2_ms": t2, "step_achieved_gbs": ach_step,
                         "algorithmic_bytes_per_cell": {"stage1": BYTES_STAGE1, "stage2": BYTES_STAGE2},
                         "limiter": "the latency of dependent FP64 operations and instruction issue, not DRAM: at "
                                    "160^3 ncu shows DRAM traffic 0.98x algorithmic, FP64 pipe 44-46 %, issue 53-54 % "
                                    "at 12 warps/SM, top stall FP64 dependency latency",
                         "fp64_pipe": {"ops_per_cell": FP64_OPS_STAGE2_PER_CELL, "achieved_tops": fp64_ach,
                                       "peak_tops": fp64_peak, "frac": fp64_ach / fp64_peak,
                                       "source": "DFMA + DMUL + DADD + DSETP thread instructions per cell of the "
                                                 "stage-2 launch (ncu at 160^3); peak 64 lanes per SM clock"}},
            "mixed": mixed,
            "c3": c3,
            "ensemble": ensemble,
            "served": served,
            "facelist": facelist,
            "cpu_baseline": base,
            "clocks": clocks,
            "gpu_launches": int(sum(k_n)),
            "diag": {"n_pfloor": diag.n_pfloor, "n_negdens": diag.n_negdens, "finite": finite},
        }
        print(json.dumps(line), flush=True)
    solver.close()
    ic_state.close()
    if world > 1:
        torch.distributed.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=256)
    ap.add_argument("--tsteps", type=int, default=200)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-mixed", action="store_true")
    ap.add_argument("--no-ensemble", action="store_true")
    ap.add_argument("--mixed-only", action="store_true")
    ap.add_argument("--mixed-precision", type=int, default=1, choices=[1, 2],
                    help="mixed form: 1 FP32 Riemann arithmetic, 2 the delta form")
    ap.add_argument("--c3", type=int, default=0, help="run config C3 (mixed vs plain) on this many seeded draws")
    ap.add_argument("--c3-n", type=int, default=384, help="C3 leg grid edge in the default line (0 = off)")
    ap.add_argument("--c3-steps", type=int, default=500)
    ap.add_argument("--c5", type=int, default=0,
                    help="run config C5 at its stated parameters (edges [32,256], cap 3000 steps, steady state "
                         "1e-5, 150 GB) on this many requests, served and sequential plain, and exit")
    ap.add_argument("--serve-requests", type=int, default=100)
    ap.add_argument("--facelist-n", type=int, default=128, help="face-list leg on an n^3 box (0 = off)")
    ap.add_argument("--serve-max-edge", type=int, default=96)
    ap.add_argument("--serve-max-steps", type=int, default=600)
    ap.add_argument("--decomp", default="replicas", choices=["replicas", "slab"],
                    help="N > 1: independent replicas (default) or one grid split along z across the ranks")
    args = ap.parse_args()
    world, rank, local = dist_setup()
    if args.impl == "reference":
        run_reference(args, world, rank)
    elif args.mixed_only:
        run_mixed_only(args)
    elif args.decomp == "slab":
        run_slab(args, world, rank, local)
    elif args.c5 > 0:
        run_c5(args)
    elif args.c3 > 0:
        import set_b200  # noqa: F401  (fails loudly without the CUDA library)
        from set_b200 import workloads as WL
        for r in WL.run_c3(WL.c3_problems(count=args.c3, n=args.n, steps=args.tsteps)):
            print(json.dumps({"leg": "C3", **r}), flush=True)
    else:
        run_ours(args, world, rank, local)


if __name__ == "__main__":
    main()
