"""Benchmark: frequency-sweep solves/s on the cylinder-in-box.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--cells 32] [--nfreq 16] [--ordering amd|nd]

One step is one sweep: the 16 log-spaced frequencies (50 Hz .. 1 MHz) of the
32^3-cell cylinder-in-box (196,608 Kuhn tets, 227,004 unknowns), each
assembled on the device (element fill + scatter), equilibrated, factorized
and solved to relative residual <= 1e-14 (the bar is 1e-10): all 16
frequencies factorized in one FP32 batch on the tensor cores, refined by
FP64 preconditioned COCG on the original systems, and any frequency whose
refinement stalls refactorized in FP64 automatically. The plain FP64
factorization of the same sweep is timed beside it (the "fp64" key). The ordering is the reference's own
AMD permutation, reproduced bit for bit on the host.

Multi-GPU: one process per GPU, each solving its own sweep (frequency
replicas, no exchange); value = solves of all ranks / max-over-ranks time.

--impl reference times the reference's own CPU implementation
(oracle/_ref, compiled from its sources) with every host core: each step is
a bounded sample of concurrent single-threaded solve_symmetric calls (one
16^3 frequency per process); ms_per_step is that step's wall time, and value
extrapolates the sample's rate to the 32^3 workload by the ratio of
factorization flops (labelled "extrapolated" in the line). Nothing of this
repository's library is loaded on that arm.
"""
from __future__ import annotations

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
sys.path.insert(0, str(ROOT / "hybrid-aphi-solver_b200"))
sys.path.insert(0, str(ROOT / "tests"))

METRIC = "solves/s & p50/p99 latency, FP32+IR vs FP64 LDLᵀ at rel. residual ≤1e-10"
UNIT = "solves/s"
F_LO, F_HI = 50.0, 1.0e6


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return d["hbm_gbs"], d["bf16_tflops"], d["bf16_tflops_sustained"], "measured"
    return 6650.0, 1590.0, 1400.0, "fallback"


class Clocks:
    """nvidia-smi samples during the timed region."""

    def __init__(self, index: int):
        self.index = index
        self.rows = []
        self.proc = None

    def __enter__(self):
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except FileNotFoundError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [x.strip() for x in line.split(",")]
            if len(parts) == 7:
                self.rows.append(parts)

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        sm = [float(r[0]) for r in self.rows if r[0].replace(".", "").isdigit()]
        mx = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in self.rows for i in range(4) if r[3 + i].lower() == "active"})
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows)}


def dist_env():
    """(rank, world size, local rank) from the launcher's environment, read
    here so that the reference arm imports nothing of the library."""
    return (int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")),
            int(os.environ.get("LOCAL_RANK", "0")))


# ---------------------------------------------------------------- CPU arm
def _ref_one(args):
    cells, omega = args
    import refbridge as rb
    r = rb.RefProblem.cylinder(cells)
    v, b = r.refill(omega)
    t0 = time.perf_counter()
    r.refill(omega)
    x, rep = r.solve_symmetric(b)
    return time.perf_counter() - t0, rep["factorize_ms"], rep["backward_error"]


def _ref_flops(cells):
    import refbridge as rb
    cc = rb.RefProblem.cylinder(cells).analysis()["col_count"].astype(np.float64) - 1.0
    return float(8.0 * np.sum(cc * (cc + 1.0) / 2.0))


def ref_flops(cells_list):
    """Factorization flops 8 * sum_j c'_j (c'_j + 1) / 2, c'_j = col_count_j - 1,
    from the reference's own AMD analysis (src/symbolic.cpp), one spawned
    process per mesh so that the large analysis's memory is returned."""
    import multiprocessing as mp
    with mp.get_context("spawn").Pool(len(cells_list)) as pool:
        return dict(zip(cells_list, pool.map(_ref_flops, cells_list)))


def host_procs(gb_per_proc: float = 0.5) -> int:
    """Concurrent reference solves for this host: one per core in the
    process's CPU affinity, capped so that they use at most half of the
    memory available (MemAvailable, or what the cgroup limit leaves);
    a 16^3 reference solve peaks near 0.35 GB."""
    cpus = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    avail = None
    try:
        with open("/proc/meminfo") as f:
            for line in f:
                if line.startswith("MemAvailable:"):
                    avail = int(line.split()[1]) * 1024
    except OSError:
        pass
    try:
        lim = Path("/sys/fs/cgroup/memory.max").read_text().strip()
        cur = int(Path("/sys/fs/cgroup/memory.current").read_text().strip())
        if lim.isdigit():
            avail = min(avail if avail is not None else 1 << 62, int(lim) - cur)
    except (OSError, ValueError):
        pass
    if avail is None:
        return cpus
    return max(1, min(cpus, int(0.5 * avail / (gb_per_proc * 2 ** 30))))


def ref_sample_step(pool, cells_sample: int, procs: int):
    """One step of the reference arm: `procs` concurrent single-threaded
    solve_symmetric calls, one sample-mesh frequency each. Returns the step's
    wall time and the slowest solve's time (s)."""
    omegas = 2 * np.pi * np.geomspace(F_LO, F_HI, procs)
    t0 = time.perf_counter()
    res = pool.map(_ref_one, [(cells_sample, om) for om in omegas], chunksize=1)
    return time.perf_counter() - t0, max(r[0] for r in res)


def extrapolation(cells_sample, cells_target, flops, per_solve_s, procs):
    ratio = flops[cells_target] / flops[cells_sample]
    rate = procs / per_solve_s / ratio
    return rate, {
        "sample_mesh": f"{cells_sample}^3 cylinder-in-box", "target_mesh": f"{cells_target}^3 cylinder-in-box",
        "sample_solves_per_s": procs / per_solve_s, "flops_ratio": ratio,
        "flops_per_factorization": {f"{c}^3": flops[c] for c in (cells_sample, cells_target)},
        "method": (f"{cells_target}^3 rate = {cells_sample}^3 rate / flop ratio, flops from the reference's own "
                   f"AMD analysis: an EXTRAPOLATION, not a {cells_target}^3 measurement. The reference's time per "
                   "flop grows with the front sizes: on one core of one machine its 32^3 factorization took "
                   "2,098 s where its 16^3 time (16.5 s) scaled by flops predicts 1,935 s, so this overstates "
                   "the reference's 32^3 rate by about 8 %")}


def cpu_reference(cells_sample: int, cells_target: int, procs: int, flops=None):
    """One bounded sample (procs concurrent sample-mesh solves), extrapolated
    to the target mesh by the factorization-flop ratio."""
    import multiprocessing as mp
    flops = flops or ref_flops([cells_sample, cells_target])
    with mp.get_context("spawn").Pool(procs) as pool:
        wall, per = ref_sample_step(pool, cells_sample, procs)
    rate, ext = extrapolation(cells_sample, cells_target, flops, per, procs)
    return {"value": rate, "unit": UNIT, "cores": procs, "kind": "reference",
            "sample": ((f"{procs} concurrent single-threaded reference solve_symmetric calls"
                        if procs > 1 else "one single-threaded reference solve_symmetric call")
                       + f" (refill + equilibrated FP64 up-looking LDL^T + solve), one {cells_sample}^3 "
                       f"frequency" + (" each" if procs > 1 else "") + f", {per:.1f} s; extrapolated to "
                       f"{cells_target}^3 by its {ext['flops_ratio']:.1f}x factorization flops"),
            "extrapolated": ext, "sample_wall_s": wall, "sample_solve_s": per}


def run_reference(args):
    """The reference's own CPU solve_symmetric (oracle/_ref, compiled from
    its sources), every host core busy. Nothing of this repository's library
    is loaded. A step is one bounded sample: one concurrent solve per core of
    a sample-mesh frequency (the 32^3 factorization takes about 35 minutes
    of one core, far beyond a step). ms_per_step is that step's measured
    wall time; value extrapolates the sample's rate to the benchmarked mesh
    and is labelled as such."""
    rank, world, _ = dist_env()
    if rank != 0:
        return
    import multiprocessing as mp
    import refbridge as rb
    if not rb.available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libaphi_ref.so was not built"}))
        return
    procs = host_procs()
    flops = ref_flops([args.sample_cells, args.cells])
    # A compiled CPU solve has nothing to warm up beyond the process pool and
    # the page cache: one untimed step, whatever --warmup says.
    walls, pers = [], []
    with mp.get_context("spawn").Pool(procs) as pool:
        ref_sample_step(pool, args.sample_cells, procs)
        for _ in range(max(args.steps, 1)):
            w, p = ref_sample_step(pool, args.sample_cells, procs)
            walls.append(w)
            pers.append(p)
    per = float(np.median(pers))
    v, ext = extrapolation(args.sample_cells, args.cells, flops, per, procs)
    base = {"value": v, "unit": UNIT, "cores": procs, "kind": "reference",
            "sample": (f"{procs} concurrent single-threaded reference solve_symmetric calls (refill + "
                       f"equilibrated FP64 up-looking LDL^T + solve), one {args.sample_cells}^3 frequency each "
                       f"per step; the rate is extrapolated to {args.cells}^3 by factorization flops"),
            "extrapolated": ext}
    out = {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
           "warmup": 1, "ms_per_step": 1000.0 * float(np.median(walls)), "higher_is_better": True,
           "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic",
           "impl": "reference",
           "config": workload_config(args, None) | {
               "timed_sample": f"{procs} concurrent {args.sample_cells}^3 frequencies per step",
               "value_is": f"extrapolated from {args.sample_cells}^3 to {args.cells}^3 by factorization flops"},
           "cpu_baseline": base,
           "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out))


def workload_config(args, info):
    cfg = {"workload": (f"cylinder-in-box {args.cells}^3 cells ({6 * args.cells ** 3} Kuhn tets), "
                        f"{args.nfreq} log-spaced frequencies {F_LO:g} Hz-{F_HI:g} Hz, reduced A-Phi, "
                        f"row_scaled, 1 V / 0 V voltage ports, {args.ordering.upper()} ordering"),
           "cells": args.cells, "frequencies": args.nfreq,
           "l2": "inputs larger than L2 (factors of several GB per frequency)"}
    if info:
        cfg.update({k: info[k] for k in ("n", "nnz_upper", "nnz_l", "supernodes", "levels", "max_rows")})
        cfg["flops_per_factorization"] = info["flops"]
    return cfg


# ---------------------------------------------------------------- GPU arm
def device_ms(fn, stream, reps=3):
    """Mean device time (ms) of fn() over reps calls after one untimed call:
    CUDA events on the stream the kernels run on, synchronized on both sides."""
    import torch
    fn()
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(stream)
    for _ in range(reps):
        fn()
    b.record(stream)
    torch.cuda.synchronize()
    return a.elapsed_time(b) / reps


def assembly_roofline(w, asm, an, nfreq, ms, hbm):
    """k_tet_terms + k_slot_sum over a whole sweep. Algorithmic
    bytes per frequency: T (16 B tet -> node ids + 96 B coordinates + 24 B edge
    ids + 6 B signs + 64 B DOF indices + 4 B body id) + 4 B per live pair of
    each tet's DOFs (its slot map, sum n_t (n_t + 1) / 2) + 16 B per stored
    value and per rhs entry written once."""
    idx = np.asarray(w.array("tet_idx")).reshape(-1, 16)
    n_t = (idx >= 0).sum(axis=1).astype(np.int64)
    T = idx.shape[0]
    per_freq = T * (16 + 96 + 24 + 6 + 64 + 4) + 4 * int(np.sum(n_t * (n_t + 1) // 2)) + 16 * (an.nnz + an.n)
    achieved = nfreq * per_freq / (ms / 1000.0) / 1e9
    # what this design moves: the term array written once and read once per
    # frequency, its slot lists read once per batch, values and rhs written
    design = nfreq * (32 * asm.num_terms + 16 * (an.nnz + an.n)) + 4 * asm.num_terms + 4 * (an.nnz + an.n)
    return {"kernels": "k_tet_terms + k_slot_sum", "bound": "hbm", "frequencies": nfreq,
            "ms_per_sweep": ms, "ms_per_frequency": ms / nfreq, "algorithmic_bytes_per_frequency": per_freq,
            "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
            "design_bytes_per_sweep": design, "design_gbs": design / (ms / 1000.0) / 1e9}


def solve_roofline(an, entries, ms, hbm):
    """FP64 forward + diagonal + backward solve of `entries` factors, one rhs
    each. Algorithmic bytes per rhs: 2 (nnz(L) - N) (16 B value + 4 B index)
    + 16 N (L read twice, y once)."""
    n, nnz_l = an.n, an.info["nnz_l"]
    per = 2 * (nnz_l - n) * (16 + 4) + 16 * n
    achieved = entries * per / (ms / 1000.0) / 1e9
    return {"kernels": "k_fwd_gather, k_fwd_diag, k_fwd_update, k_bwd_update, k_bwd_diag (FP64)",
            "bound": "hbm", "entries": entries, "ms": ms, "algorithmic_bytes_per_rhs": per,
            "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm}


def parity_vs_reference(args, rank, omegas, x):
    """Per fixture frequency: ||x - x_ref|| / ||x_ref|| against the
    reference's own solve_symmetric solution of the same system."""
    try:
        import reference_solutions as refsol
    except ImportError:
        return None
    fx = refsol.load(args.cells) if rank == 0 else None
    if fx is None:
        return None
    out = []
    for j, k in enumerate(fx["sweep_index"]):
        if k >= len(omegas) or omegas[k] != fx["omegas"][j]:
            continue
        xk = x[k].cpu().numpy()
        xr = fx["x"][j]
        out.append({"f_hz": float(omegas[k] / (2 * np.pi)), "sweep_index": int(k),
                    "rel_diff_vs_reference": float(np.linalg.norm(xk - xr) / np.linalg.norm(xr)),
                    "reference_rel_residual": fx["reports"][j]["residual"]})
    return {"fixture": refsol.path(args.cells).name,
            "note": ("the reference's own FP64 solution is itself off the exact one by ~2e-12 at 50 Hz, "
                     "~3e-10 at 10 kHz and ~1e-8 at 1 MHz (cond grows with frequency); tests/"
                     "test_headline_parity_gpu.py checks these against an extended-precision solution"),
            "frequencies": out}


def update_kernel(precision, kind, tc_split, live):
    """The kernel that serves a kind of update, the peak of its useful flops
    [TFLOP/s] and what that is. The INT8 tiles form 36 (FP64: eight digits,
    eight levels) or 10 (FP32: four and four) digit products per real product,
    at a peak of four times the TF32 one (the nominal ratio)."""
    digits = {"fp64": 36, "fp32": 10}[precision]
    int8 = (4.0 * live["tf32_tc_n256"] / digits, f"4 x tf32_tc_n256 / {digits} digit products")
    if kind == "update_tc":
        if tc_split == 2 and "APHI_TC_PRESPLIT" not in os.environ:
            return ("k_update_i8<float> (tcgen05 INT8-digit trailing update)", *int8)
        return "k_update_tc (tcgen05 split-TF32 trailing update)", live["tf32_tc_n256"], "tf32_tc_n256"
    if precision == "fp32":
        return (f"k_update_wide<float> (SIMT {kind})" if kind == "update_wide" else kind), live["fp32_ffma"], "fp32_ffma"
    if kind == "update_wide" and os.environ.get("APHI_DMMA_PRESCALE") != "0":
        return ("k_update_i8<double> (tcgen05 INT8-digit trailing update)", *int8)
    return f"k_update_wide_dmma (FP64 DMMA {kind})", live["fp64_dmma"], "fp64_dmma"


def run_ours(args):
    import torch
    import aphi_b200 as ab

    rank, world, local = dist_env()
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600), device_id=dev)

    from aphi_b200 import replicas
    barrier = replicas.barrier

    # Host-side per-mesh setup (untimed, once): workload, ordering, analysis.
    w = ab.Workload.cylinder(args.cells)
    if args.ordering == "amd":
        perm = ab.amd_ordering(w.row_ptr, w.col_idx)
    else:
        perm = ab.nested_dissection(w.row_ptr, w.col_idx, w.dof_xyz)
    asm = ab.Assembly(ab.workload_arrays(w))
    # Each rank solves its own sweep: the frequencies shifted per rank.
    omegas = replicas.rank_omegas(rank, args.nfreq, F_LO, F_HI)
    tune_record = None
    if args.autotune:
        # The schedule's knobs (panel groups, one-CTA fronts) tuned on this
        # mesh by timed factorizations of two of the sweep's frequencies, in
        # both precisions, weighted by how many entries each precision takes.
        from aphi_b200 import autotune
        tv, _ = asm.refill(omegas[[0, -1]])
        an, tune_record = autotune.tune(w.row_ptr, w.col_idx, perm, tv, precisions=(ab.PREC_FP64, ab.PREC_FP32),
                                        weights={ab.PREC_FP64: 9.0, ab.PREC_FP32: 7.0})
        del tv
        torch.cuda.empty_cache()
    else:
        an = ab.Analysis(w.row_ptr, w.col_idx, perm)
    info = an.info
    n = an.n
    stream = torch.cuda.current_stream()

    solver = ab.SweepSolver(an, asm, args.nfreq, "mixed", fp64_batch=args.fp64_batch, rtol=args.rtol,
                            tol=args.tol, tc_split=args.tc_split, fp32_batch=args.fp32_batch or None)
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731

    def sweep():
        return solver.solve(omegas, stream=stream)

    for _ in range(args.warmup):
        sweep()
    torch.cuda.synchronize()
    live_peaks = ab.measure_peaks()
    barrier()
    torch.cuda.synchronize()
    launches0 = ab.launch_count()
    # Per-kind device time of the factorizations inside the timed steps: CUDA
    # events around each launch, on the stream the kernels run on.
    # Only the trailing-update kinds are timed (two events per launch): the
    # roofline needs the dominant kernel's durations, and fewer events
    # perturb the timed sweep less.
    solver.profile(True, kinds=("update_wide", "update_tc", "update_panel"))
    step_ms = []
    torch.cuda.nvtx.range_push("timed")   # ncu --nvtx --nvtx-include "timed/" captures exactly these steps
    with Clocks(local) as clk:
        t0, t1 = ev(), ev()
        t0.record(stream)
        for _ in range(args.steps):
            s0, s1 = ev(), ev()
            s0.record(stream)
            x, vals, rhs, reps = sweep()
            s1.record(stream)
            torch.cuda.synchronize()
            step_ms.append(s0.elapsed_time(s1))
        t1.record(stream)
        torch.cuda.synchronize()
        barrier()
    torch.cuda.nvtx.range_pop()
    launches = (ab.launch_count() - launches0) // max(args.steps, 1)
    kind_ms = solver.profile_read()
    entries = {"fp32": solver.factorized[ab.PREC_FP32], "fp64": solver.factorized[ab.PREC_FP64]}
    solver.profile(False)
    elapsed = t0.elapsed_time(t1)   # this rank's; the job's is the slowest rank's (below)
    res = ab.residuals(an, vals, x, rhs)

    # The dominant kernel of the timed steps and its roofline: useful
    # Schur-update flops (lower-triangle entries of the fronts, 8 real flops
    # per complex multiply-add) of every factorization it served, over its
    # summed launch durations.
    plan_flops = {"fp32": an.plan_stats(1, flops=True), "fp64": an.plan_stats(0, flops=True)}
    kernels = []
    for prec, kinds in kind_ms.items():
        for kind, (n_launch, ms) in kinds.items():
            st = plan_flops[prec].get(kind)
            useful = st[2] * entries[prec] if st else 0.0
            kernels.append({"precision": prec, "kind": kind, "launches": n_launch, "ms": ms,
                            "share_of_step": ms / elapsed, "useful_tflop": useful / 1e12,
                            "tflops": useful / (ms / 1000.0) / 1e12 if useful else None})
    kernels.sort(key=lambda k: -k["ms"])
    top = kernels[0]
    name, peak, peak_source = update_kernel(top["precision"], top["kind"], args.tc_split, live_peaks)

    # The timed sweep's solutions against the reference's own solutions of
    # the same systems, where a fixture of this mesh exists (rank 0 solves the
    # unshifted sweep; tests/golden/make_reference_solutions.py wrote them).
    parity = parity_vs_reference(args, rank, omegas, x)

    # End to end through the reference-facing calls with host buffers: refill
    # hands the assembled systems to the host (as refill(SymmetricSystem&)
    # does), solve_symmetric takes them back with the right-hand sides and
    # returns the solutions to the host.
    host_vals = torch.empty((args.nfreq, an.nnz), dtype=torch.complex128, pin_memory=True)
    host_rhs = torch.empty((args.nfreq, n), dtype=torch.complex128, pin_memory=True)
    host_x = torch.empty((args.nfreq, n), dtype=torch.complex128, pin_memory=True)
    dvals = torch.empty((args.nfreq, an.nnz), dtype=torch.complex128, device=dev)
    drhs = torch.empty((args.nfreq, n), dtype=torch.complex128, device=dev)

    def e2e_step():
        v, r = asm.refill(omegas, stream=stream)
        host_vals.copy_(v, non_blocking=True)
        host_rhs.copy_(r, non_blocking=True)
        dvals.copy_(host_vals, non_blocking=True)
        drhs.copy_(host_rhs, non_blocking=True)
        xx, _, _, _ = solver.solve(omegas, stream=stream, values=dvals, rhs=drhs)
        host_x.copy_(xx, non_blocking=True)

    e2e_step()
    torch.cuda.synchronize()
    barrier()
    a, b = ev(), ev()
    a.record(stream)
    for _ in range(args.steps):
        e2e_step()
    b.record(stream)
    torch.cuda.synchronize()
    barrier()
    e2e_ms = a.elapsed_time(b) / args.steps
    h2d = 2 * (host_vals.numel() + host_rhs.numel()) * 8
    d2h = 2 * (host_vals.numel() + host_rhs.numel() + host_x.numel()) * 8

    solver.close()
    del solver
    torch.cuda.empty_cache()

    # Plain FP64 factorization of the same sweep (the drop-in path).
    fp64 = ab.SweepSolver(an, asm, args.nfreq, "fp64", fp64_batch=args.fp64_batch)
    fp64.solve(omegas, stream=stream)
    torch.cuda.synchronize()
    barrier()
    a, b = ev(), ev()
    a.record(stream)
    for _ in range(args.fp64_steps):
        x64, vals64, rhs64, _ = fp64.solve(omegas, stream=stream)
    b.record(stream)
    torch.cuda.synchronize()
    barrier()
    fp64_ms = a.elapsed_time(b) / args.fp64_steps
    res64 = ab.residuals(an, vals64, x64, rhs64)

    # The job's figures are the slowest rank's: one max-over-ranks reduction.
    elapsed, e2e_ms, fp64_ms = replicas.max_over_ranks([elapsed, e2e_ms, fp64_ms], device=dev)
    value = replicas.job_rate(world, args.nfreq * args.steps, elapsed)
    e2e_value = replicas.job_rate(world, args.nfreq, e2e_ms)
    fp64_value = replicas.job_rate(world, args.nfreq, fp64_ms)
    # The HBM-bound parts on their own, device-resident: the assembly (element
    # fill + scatter, all frequencies of the sweep in one batch) and the FP64
    # triangular solves of one factor batch.
    asm_ms = device_ms(lambda: asm.refill(omegas, stream=stream), stream, reps=5)
    f64 = fp64.f64
    b64 = rhs64[args.nfreq - f64.batch:].contiguous()   # the entries the resident factor holds
    solve_ms = device_ms(lambda: f64.solve(b64, stream=stream), stream, reps=3)
    if_hbm = peaks()[0]
    assembly_line = assembly_roofline(w, asm, an, args.nfreq, asm_ms, if_hbm)
    solve_line = solve_roofline(an, f64.batch, solve_ms, if_hbm)
    fp64.close()
    del fp64

    hbm, bf16, bf16s, src = peaks()
    # DRAM traffic of the dominant kernel: only three launches at 24^3 have been
    # captured (a capture of the whole factorization at this size is too large).
    traffic = None
    traffic_note = "not captured at this size; three launches at 24^3 in profiles/k_update_i8_cylinder24.md"
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu:
        try:
            import refbridge as rb
            if rb.available():
                cpu = cpu_reference(args.sample_cells, args.cells, 1)
        except Exception as e:  # the baseline is reported, not required
            cpu = {"unavailable": str(e)}

    if rank == 0:
        out = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": elapsed / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None,
            "dtype": "c64 or c128 factor, c128 refinement", "data": "synthetic",
            "config": workload_config(args, info) | {"batch": args.nfreq, "parallelism": f"freq-replicas x{world}"},
            "latency_ms": {"p50": float(np.percentile(step_ms, 50)), "p99": float(np.percentile(step_ms, 99)),
                           "what": "one sweep of all frequencies (every solve of the batch completes together)"},
            "accuracy": {"max_backward_error": float(res[..., 1].max()), "max_rel_residual": float(res[..., 0].max()),
                         "fp32_entries": sum(r["precision"] == "fp32" for r in reps),
                         "fp64_entries": sum(r["precision"] == "fp64" for r in reps),
                         "fp64_predicted_entries": sum(r["predicted_fp64"] for r in reps),
                         "cocg_iterations": [r["iterations"] for r in reps]},
            "fp64": {"value": fp64_value, "unit": UNIT, "ms_per_sweep": fp64_ms, "batch": args.fp64_batch,
                     "max_rel_residual": float(res64[..., 0].max()),
                     "max_backward_error": float(res64[..., 1].max())},
            "speedup_vs_fp64": value / fp64_value,
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h)},
            "roofline": {"bound": "tensor", "kernel": name, "achieved": top["tflops"],
                         "peak": peak, "unit": "TFLOP/s", "frac": top["tflops"] / peak,
                         "peak_source": (f"{peak_source}, measured live on this device by aphi_measure_peaks "
                                         f"(the file of measured peaks has only HBM and bf16: bf16 {bf16:.0f} TF/s, {src})"),
                         "traffic": traffic, "traffic_method": traffic_note,
                         "algorithmic": (f"useful Schur-update flops: {plan_flops[top['precision']][top['kind']][2]:.4e} "
                                         f"per factorization x {entries[top['precision']]} factorizations in the "
                                         f"timed steps"),
                         "launches": top["launches"], "kernel_ms": top["ms"]},
            "kernels": kernels[:8],
            "live_peaks_tflops": live_peaks,
            "cpu_baseline": cpu,
            "gpu_launches": int(launches),
            "clocks": clk.summary(),
            "assembly_roofline": assembly_line,
            "solve_roofline": solve_line,
            "parity_vs_reference": parity,
            "autotune": tune_record,
        }
        print(json.dumps(out))
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cells", type=int, default=32)
    ap.add_argument("--nfreq", type=int, default=16)
    ap.add_argument("--ordering", default="amd", choices=["amd", "nd"])
    ap.add_argument("--tol", type=float, default=1e-16, help="backward-error target of the refinement")
    ap.add_argument("--rtol", type=float, default=1e-14,
                    help="relative-residual target of the refinement (the FP64 direct solve's own level)")
    ap.add_argument("--fp64-batch", type=int, default=8)
    ap.add_argument("--fp32-batch", type=int, default=0, help="FP32 entries per factorization (0: the whole sweep)")
    ap.add_argument("--tc-split", type=int, default=2, choices=[2, 3],
                    help="the FP32 tensor-core update's form (2: INT8 digits; 3: three TF32 pieces per operand)")
    ap.add_argument("--fp64-steps", type=int, default=1)
    ap.add_argument("--sample-cells", type=int, default=16)
    ap.add_argument("--autotune", type=int, default=1, help="tune the schedule on this mesh first (untimed)")
    ap.add_argument("--no-cpu", action="store_true")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
