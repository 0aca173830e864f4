"""Benchmark of the fixed-effects solve on B200.

Workload (N = 1): the 10,000,000-row worker/firm/year panel (1,000,000
workers, 100,000 Pareto(1.5) firms, 20 years; seeded synthetic data, see
within_b200/workloads.py), y ~ N(0,1), default additive Schwarz, tol 1e-8.
A step is one full solve (Solver::solve with the preconditioner reused)
of one right-hand side.  ``value`` is whole-job solves/s with y already in
HBM; ``e2e`` is the same through the public host API (y copied in, demeaned and
x copied out every step).  The working set (codes, permutations and vectors,
> 500 MB) exceeds the 126 MB L2, so no explicit flush is needed.

Multi-GPU (torchrun): replicas only -- every rank solves its own copy of the
workload with no collective on the data path; timing is the max over ranks.

``--impl reference`` times the reference algorithm's CPU restatement
(oracle/, the reference itself cannot be built here: no Rust toolchain) on the
host cores, on rank 0 only.
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

METRIC = "solve time & HBM GB/s at 1e-8; mixed/batched vs plain GPU LSMR, same accuracy"
UNIT = "solves/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--rows", type=int, default=10_000_000)
    ap.add_argument("--tol", type=float, default=1e-8)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-mixed", action="store_true", help="skip the mixed-precision batched section")
    ap.add_argument("--no-many", action="store_true", help="skip the many-designs section")
    ap.add_argument("--many", type=int, default=256, help="designs in the many-designs section")
    ap.add_argument("--no-autograd", action="store_true", help="skip the differentiable-demeaning section")
    ap.add_argument("--no-published", action="store_true",
                    help="skip the reference's published 1M-row wall-clock configuration")
    ap.add_argument("--kernel-timeline", choices=["fp64", "mixed"], default=None,
                    help="instead of the bench line: per-kernel device times of one solve (torch.profiler "
                         "/ CUPTI timestamps); 'mixed' = weighted panel, k = 4, mixed precision")
    ap.add_argument("--setup-trace", action="store_true",
                    help="instead of the bench line: Solver::new + first solve (best of 3) of the fixest-like "
                         "1M design and the 10M panel, each in its own process, with the set-up's phase "
                         "trace (WITHIN_TRACE=1) of the best run")
    ap.add_argument("--tuning", default="auto",
                    help="tuning record of the headline solver: 'auto' (the autotuner's table), 'none' (the "
                         "defaults and WITHIN_* overrides) or a JSON dict of within_tuning fields")
    ap.add_argument("--cpu-sample-iters", type=int, default=3)
    ap.add_argument("--ref-budget-s", type=float, default=150.0,
                    help="host seconds the reference arm's warm-up and timed steps may take before each "
                         "step becomes a bounded run of iterations")
    return ap.parse_args()


# DRAM bytes (dram__bytes_read.sum + dram__bytes_write.sum) per launch of the
# design-operator pair's kernels, from one ncu capture (--clock-control none)
# of the 4,000,000-row panel: the staged gather k_tgather<3,0,0> (D x) and the
# staged adjoint sweep k_tsweep<1,0,3,2,1,0,0> with its crossing-run fix-up
# k_rw_fix<1,0> and the run combine k_seglist<SlScatter<1>> (D^T u).  Every stream of the pair grows with the row count on this panel
# generator (workers n/10, firms n/100), so a 10,000,000-row launch moves 2.5x.
PAIR_TRAFFIC_4M = {"gather": 51_707_904, "adjoint": 90_450_944}
PAIR_TRAFFIC_KERNELS = "k_tgather<3,0,0> + k_tsweep<1,0,3,2,1,0,0> + k_rw_fix<1,0> + k_seglist<SlScatter<1>>"


def pair_traffic(n, q, solver):
    """The pair's DRAM bytes per launch (gather + adjoint) scaled from the 4M-row
    capture, or None when the workload or the kernels differ from the capture's."""
    t = solver.tuning
    if t is None:
        staged = os.environ.get("WITHIN_TSWEEP", "1") != "0" and os.environ.get("WITHIN_SWEEP", "2") != "0"
        ranges = int(os.environ.get("WITHIN_WARP_RANGES", "1"))
    else:
        staged, ranges = t.get("staged_sweep", 1) == 1, t.get("warp_ranges", 1)
    if q != 3 or not staged or ranges != 1:
        return None, None
    f = n / 4_000_000
    return (f * (PAIR_TRAFFIC_4M["gather"] + PAIR_TRAFFIC_4M["adjoint"]),
            f"ncu capture of the 4,000,000-row panel x {f:g}: {PAIR_TRAFFIC_KERNELS}")


def tuning_arg(args):
    t = getattr(args, "tuning", "auto")
    if t == "auto":
        return "auto"
    if t == "none":
        return None
    return json.loads(t)


def workload(rows):
    from within_b200 import workloads as W
    workers = max(1, rows // 10)
    firms = max(1, rows // 100)
    codes = W.akm_panel(n=rows, n_workers=workers, n_firms=firms)
    y = W.akm_response(rows)
    return codes, y


def config_dict(rows, n_dofs=None):
    return {
        "workload": f"akm panel n={rows} (worker {rows // 10}, firm {rows // 100} Pareto(1.5), year 20), "
                    "1 RHS, default additive Schwarz, tol 1e-8",
        "n_obs": rows, "n_dofs": n_dofs, "k_rhs": 1, "precision": "fp64",
        "l2_policy": "working set > L2 (no flush)", "parallelism": "replicas",
    }


class Clocks:
    """nvidia-smi sampler running during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.rows = []
        self._stop = threading.Event()
        self._t = None

    def _run(self):
        while not self._stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                      "--format=csv,noheader,nounits"], capture_output=True, text=True,
                                     timeout=5).stdout.strip()
                if out:
                    self.rows.append([c.strip() for c in out.split(",")])
            except Exception:
                pass
            self._stop.wait(0.2)

    def __enter__(self):
        self._t = threading.Thread(target=self._run, daemon=True)
        self._t.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        self._t.join(timeout=10)

    def summary(self):
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            for name, v in zip(names, r[5:9]):
                if v.strip().lower() == "active":
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(self.rows)}


def peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def demeaned_err(D, Dref, Y):
    """max|D - Dref| per column, scaled by max|y| ("inf_over_inf") and by
    ||y||_2 ("inf_over_l2", the scaling the 1e-7 contract is stated in); the
    worst column of each."""
    D = D.reshape(D.shape[0], -1)
    Dref = Dref.reshape(Dref.shape[0], -1)
    Y = Y.reshape(Y.shape[0], -1)
    d = (D - Dref).abs().max(dim=0).values
    return {"inf_over_inf": float((d / Y.abs().max(dim=0).values).max()),
            "inf_over_l2": float((d / Y.norm(dim=0)).max())}


def iteration_bytes(n, nd, Q, k=1, s=8, weighted=False, n_slopes=0, ps=None):
    """Algorithmic bytes of one LSMR iteration of k columns (value size s):
    - op_survey: the design-operator pair as a gather pass plus a scatter pass,
      2 (4 n Q + s n S + s n [w]) + s n (1 + 2k) + s n_dofs 2k;
    - op_fused: the same with the codes, loadings and sqrt(w) read once (the
      fused row sweep): 4 n Q + s n S + s n [w] + 2 s n k + 2 s n_dofs k;
    - precond: every preconditioner non-zero read with its column index and
      the vector entry it multiplies ((4 + 2s) each: C, C^T, factor, dense
      blocks and cores), plus restrict / means / prolongation over the local
      slots (4 + 5s each) and the output (s n_dofs), times k;
    - vectors: 15 s n_dofs k (p~ update, alpha dot, v scale, solution update)."""
    w = 1 if weighted else 0
    op_survey = 2 * (4 * n * Q + s * n * n_slopes + s * n * w) + s * n * (1 + 2 * k) + s * nd * 2 * k
    op_fused = 4 * n * Q + s * n * n_slopes + s * n * w + 2 * s * n * k + 2 * s * nd * k
    pm = 0
    if ps and ps.get("n_subdomains"):
        nnz = ps["nnz_c"] + ps["nnz_ct"] + ps["nnz_fwd"] + ps["nnz_bwd"] + ps["nnz_dense"] + ps["nnz_core"]
        pm = k * (nnz * (4 + 2 * s) + ps["n_slots"] * (4 + 5 * s) + s * nd)
    elif ps:
        pm = k * 3 * s * nd
    return {"op_survey": op_survey, "op_fused": op_fused, "precond": pm, "vectors": 15 * s * nd * k}


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def max_over_ranks(value, world, device=None):
    if world == 1:
        return value
    import torch
    import torch.distributed as dist
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


# ---------------------------------------------------------------------------
def cpu_baseline(codes, y, tol, sample_iters):
    """The oracle (CPU restatement) on the same design: build once, then time
    `sample_iters` LSMR iterations and scale to the iteration count of a full
    solve measured on a bounded run."""
    from oracle import oracle as O
    O.build()
    threads = os.cpu_count() or 1
    O.lib().or_set_threads(threads)
    t0 = time.perf_counter()
    s = O.OracleSolver(codes)
    t_setup = time.perf_counter() - t0
    t1 = time.perf_counter()
    r = s.solve(y, tol=tol, maxiter=sample_iters)
    t_iter = (time.perf_counter() - t1) / max(1, r.iterations)
    return s, t_setup, t_iter


def run_reference(args):
    """The reference's CPU path (the C++ restatement on every host thread) on
    the same workload: one untimed full solve gives the converged iteration
    count, then W - 1 more warm-up steps and K timed steps.  A step is a full
    solve when (K + W - 1) of them fit --ref-budget-s, else a bounded run of m
    LSMR iterations scaled to the full count (solve time per iteration is
    constant: every iteration applies the same operator and preconditioner)."""
    rank, world, local = dist_env()
    if rank != 0:
        return
    codes, y = workload(args.rows)
    s, t_setup, t_iter = cpu_baseline(codes, y, args.tol, args.cpu_sample_iters)
    # iterations of a full solve: the GPU path's count for the same design
    # would differ (its approximate factor differs); use the restatement's own
    # converged count on this design.
    r0 = s.solve(y, tol=args.tol, maxiter=1000)
    n_it = max(1, r0.iterations)
    steps, more_warm = max(1, args.steps), max(0, args.warmup - 1)
    budget = args.ref_budget_s
    full = (steps + more_warm) * r0.time_solve <= budget
    per_it = max(t_iter, r0.time_solve / n_it)
    m = 1000 if full else max(1, min(n_it, int(budget / ((steps + more_warm) * per_it))))
    for _ in range(more_warm):
        s.solve(y, tol=args.tol, maxiter=m)
    t_steps = []
    for _ in range(steps):
        r = s.solve(y, tol=args.tol, maxiter=m)
        t_steps.append(r.time_solve * (n_it / max(1, r.iterations)))
    t_solve = sum(t_steps) / steps
    value = 1.0 / t_solve
    cores = os.cpu_count() or 1
    what = "one full solve" if full else f"{m} of the {n_it} LSMR iterations of a full solve (scaled)"
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": steps,
        "warmup": args.warmup, "ms_per_step": t_solve * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic", "impl": "reference",
        "config": config_dict(args.rows, s.n_dofs),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"per step {what} of the same design by the C++ restatement "
                                   f"({cores} host threads: row loops, reductions, SpMVs and the "
                                   f"subdomains split over threads; setup {t_setup:.1f}s excluded; "
                                   f"full solve {n_it} iterations, converged={r0.converged}); "
                                   f"host has {cores} cores"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def mixed_section(W, codes, dev, stream, args):
    """Mixed precision against plain FP64 at the same batch width and the same
    accuracy: the weighted variant of the panel (weights lognormal(0, 1)),
    k = 4 right-hand sides through one multi-RHS solve on both arms (a plain
    FP64 Solver and a mixed-precision Solver of the same design), at tol 1e-8
    (the contract tolerance) and at tol 1e-11, where the plain solve is within
    1e-8 of the FP64 solve at tol 1e-12 in max|d| / max|y| -- the accuracy the
    target compares at.  Errors of both arms in both scalings; the arms are
    timed in alternating rounds (medians) so that a transient slowdown of the
    shared machine does not land on one arm only."""
    import torch
    n = codes.shape[0]
    rng = np.random.default_rng(4)
    w = rng.lognormal(0.0, 1.0, n)
    k = 4
    Y = torch.tensor(np.asfortranarray(rng.standard_normal((n, k))), device=dev).t().contiguous().t()
    s = W.Solver(codes, weights=w, device=dev.index)
    sm = W.Solver(codes, weights=w, device=dev.index, precision="mixed")
    _, Dref, _ = s.solve_device(Y, W.LsmrOptions(tol=1e-12, maxiter=20000))

    def timed(fn, reps):
        fn()
        torch.cuda.synchronize(dev)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        for _ in range(reps):
            out = fn()
        b.record(stream)
        torch.cuda.synchronize(dev)
        return a.elapsed_time(b) / 1e3 / reps, out

    reps = max(2, args.steps // 3)
    out = {"k": k, "weights": "lognormal(0,1)", "unit": UNIT,
           "note": "errors: max|demeaned - FP64 tol 1e-12 demeaned| per column, worst column, over max|y| "
                   "(inf_over_inf) and over ||y||_2 (inf_over_l2)"}
    for tol in (args.tol, 1e-11):
        opts = W.LsmrOptions(tol=tol, maxiter=20000)
        for _ in range(2):
            s.solve_device(Y, opts)
            sm.solve_device(Y, opts)
        rp, rm = [], []
        for _ in range(4):
            tp, (_, Dp, stp) = timed(lambda: s.solve_device(Y, opts), reps)
            tm, (_, Dm, stm) = timed(lambda: sm.solve_device(Y, opts), reps)
            rp.append(tp)
            rm.append(tm)
        tpm, tmm = float(np.median(rp)), float(np.median(rm))
        out[f"tol_{tol:g}"] = {
            "plain_fp64_k4": {"value": k / tpm, "ms_per_batch": tpm * 1e3, "iterations": [x[1] for x in stp],
                              "err": demeaned_err(Dp, Dref, Y)},
            "mixed_k4": {"value": k / tmm, "ms_per_batch": tmm * 1e3, "iterations": [x[1] for x in stm],
                         "converged": all(x[0] for x in stm), "err": demeaned_err(Dm, Dref, Y)},
            "speedup_mixed_vs_plain": tpm / tmm,
            "rounds_ms": {"plain": [round(1e3 * t, 3) for t in rp], "mixed": [round(1e3 * t, 3) for t in rm]}}
    acc = out["tol_1e-11"]
    out["value"] = acc["mixed_k4"]["value"]
    out["target"] = {"accuracy": "both arms <= 1e-8 (inf_over_inf) at tol 1e-11",
                     "met_accuracy": acc["plain_fp64_k4"]["err"]["inf_over_inf"] <= 1e-8 and
                     acc["mixed_k4"]["err"]["inf_over_inf"] <= 1e-8,
                     "speedup": acc["speedup_mixed_vs_plain"], "speedup_target": 2.0}
    del s, sm
    return out


def published_section(W, args):
    """The reference's one published measurement (benches/wallclock_reference.json:5,
    crates/within/benches/wallclock_1m3fe.rs:21-50): best of 5 wall-clock runs
    of Solver::new + solve on the 1,000,000-row fixest-like panel with three
    fixed effects (10 observations per worker, 10 years, firm = i % n_firm,
    crates/within/benches/shared/fixest_dgp.rs:13-62), y uniform(-1, 1), tol
    1e-6, maxiter 200, default additive Schwarz: 170.905 ms on a GitHub
    Actions runner.  Here the timer also covers the design build (locality
    sort), which the reference builds before its timer, and host numpy y in,
    demeaned and x out; the oracle (C++ restatement, every host thread) runs
    the same sequence."""
    from within_b200 import workloads as WL
    codes, y = WL.fixest_like()
    opts = W.LsmrOptions(tol=1e-6, maxiter=200)
    runs = []
    for _ in range(5):
        t0 = time.perf_counter()
        s = W.Solver(codes)
        t1 = time.perf_counter()
        r = s.solve(y, opts)
        t2 = time.perf_counter()
        runs.append((t2 - t0, t1 - t0, t2 - t1, r.iterations, r.converged))
        del s
    best = min(runs, key=lambda x: x[0])
    out = {"workload": "fixest-like 1,000,000 x 3 FE (indiv 100,000, year 10, firm 4,348 = i % n_firm), "
                       "tol 1e-6, maxiter 200", "best_of": 5, "best_ms": best[0] * 1e3,
           "setup_ms": best[1] * 1e3, "solve_ms": best[2] * 1e3, "iterations": best[3], "converged": best[4],
           "all_ms": [round(x[0] * 1e3, 3) for x in runs], "reference_published_ms": 170.905,
           "reference_published_hardware": "GitHub Actions ubuntu-latest runner (core count not recorded)"}
    if not args.no_cpu_baseline:
        try:
            from oracle import oracle as O
            O.build()
            O.lib().or_set_threads(os.cpu_count() or 1)
            orr = []
            for _ in range(3):
                t0 = time.perf_counter()
                so = O.OracleSolver(codes)
                ro = so.solve(y, tol=1e-6, maxiter=200)
                orr.append((time.perf_counter() - t0, ro.iterations))
                del so
            ob = min(orr)
            out["cpu_restatement"] = {"best_ms": ob[0] * 1e3, "best_of": 3, "iterations": ob[1],
                                      "cores": os.cpu_count() or 1, "kind": "port"}
        except Exception as e:  # the baseline must not sink the GPU line
            out["cpu_restatement"] = {"failed": str(e)}
    return out


def many_device_time(W, ss, Yd, opts, threads=8):
    """Device time of one batch over every design of `ss` with inputs and
    outputs resident: `threads` host threads, each driving its designs on its
    own stream through within_solver_solve_batch_device; the batch time is
    the latest stream's end event against one start event all streams wait
    on (the device clock)."""
    import ctypes as C
    import torch
    from within_b200 import _ffi
    L = _ffi.lib()
    n = len(ss._h)
    Xd = [torch.empty((Y.shape[1], nd), dtype=torch.float64, device=Y.device).t()
          for Y, nd in zip(Yd, ss._n_dofs)]
    Dd = [torch.empty((Y.shape[1], Y.shape[0]), dtype=torch.float64, device=Y.device).t() for Y in Yd]
    streams = [torch.cuda.Stream() for _ in range(threads)]
    oc = opts._c()
    errs = []

    def run_once():
        start = torch.cuda.Event(enable_timing=True)
        ends = [torch.cuda.Event(enable_timing=True) for _ in streams]
        torch.cuda.synchronize()
        start.record()
        for st in streams:
            st.wait_event(start)

        def work(t):
            try:
                for i in range(t, n, threads):
                    k = Yd[i].shape[1]
                    stats = (_ffi.SolveStatsC * k)()
                    _ffi.check(L.within_solver_solve_batch_device(
                        ss._h[i], C.c_void_p(Yd[i].data_ptr()), k, C.byref(oc), C.c_void_p(Xd[i].data_ptr()),
                        C.c_void_p(Dd[i].data_ptr()), stats, C.c_void_p(streams[t].cuda_stream)))
                ends[t].record(streams[t])
            except Exception as e:   # reported after the join
                errs.append(e)
        th = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
        for x in th:
            x.start()
        for x in th:
            x.join()
        torch.cuda.synchronize()
        if errs:
            raise errs[0]
        return max(start.elapsed_time(e) for e in ends) / 1e3

    run_once()
    return float(np.median([run_once() for _ in range(3)]))


def many_section(W, args):
    """Many independent designs: `args.many` designs with n log-uniform in
    [1e4, 2e6], 2-3 uniform factors with level counts log-uniform in
    [20, n/10], k = 8 right-hand sides each, through SolverSet.solve_batch
    (host buffers in and out); solves/s = designs x 8 / wall time of the
    batch (host-driven concurrent streams, so the host clock is the measure)."""
    from within_b200 import workloads as WL
    cases = WL.many_designs(count=args.many, k=8)
    rows = int(sum(c.shape[0] for c, _ in cases))
    t0 = time.perf_counter()
    ss = W.SolverSet([c for c, _ in cases], threads=16)
    t_setup = time.perf_counter() - t0
    Ys = [Y for _, Y in cases]
    opts = W.LsmrOptions(tol=args.tol)
    res = {"designs": len(cases), "k": 8, "rows_total": rows, "unit": UNIT, "setup_s": t_setup,
           "timing": "host wall clock of SolverSet.solve_batch (median of 3), host buffers in and out; "
                     "device_value: the device clock of the same batch with inputs and outputs resident "
                     "(8 host threads, one stream each, median of 3)"}
    import torch
    Yd = [torch.tensor(np.asfortranarray(Y), device="cuda").t().contiguous().t() for Y in Ys]
    ref = None
    for prec in ("fp64", "mixed"):
        ss.set_precision(prec)
        out = ss.solve_batch(Ys, opts, want_x=False)
        ts = []
        for _ in range(3):
            t1 = time.perf_counter()
            out = ss.solve_batch(Ys, opts, want_x=False)
            ts.append(time.perf_counter() - t1)
        t = float(np.median(ts))
        its = [it for o in out for it in o[3]]
        r = {"value": len(cases) * 8 / t, "s_per_batch": t, "iterations_max": int(max(its)),
             "iterations_median": float(np.median(its)), "converged": all(all(o[2]) for o in out)}
        td = many_device_time(W, ss, Yd, opts)
        r["device_value"] = len(cases) * 8 / td
        r["device_s_per_batch"] = td
        if ref is None:
            ref = [o[1] for o in out]
        else:   # mixed against the FP64 arm at the same tolerance, worst design and column
            r["max_abs_diff_vs_fp64_over_max_y"] = max(
                float(np.max(np.abs(o[1] - d0)) / max(np.max(np.abs(Y)), 1e-300)) for o, d0, Y in zip(out, ref, Ys))
        res[prec] = r
    res["value"] = res["fp64"]["value"]
    del Yd
    del ss
    return res


def autograd_section(W, dev):
    """Differentiable demeaning on the varying-slopes panel (n = 2e6, firm 50k
    Pareto(1.5) with intercept + slope, year 30, weights lognormal(0, 0.5)):
    forward and backward time, and the gradients against central differences
    (step 1e-6) of the GPU solver on 64 weight and 64 response coordinates."""
    import torch
    from within_b200 import workloads as WL
    firm, year, x, z, w, v = WL.slopes_panel()
    eff = [W.Effect(firm, True, [x]), W.Effect(year, True)]
    opts = W.LsmrOptions(tol=1e-13, maxiter=20000)
    zt = torch.tensor(z, device=dev, requires_grad=True)
    wt = torch.tensor(w, device=dev, requires_grad=True)
    vt = torch.tensor(v, device=dev)
    solver = W.Solver(eff, weights=w, device=dev.index)
    out = W.demean(zt, eff, weights=wt, options=opts, solver=solver)
    (vt * out).sum().backward()
    torch.cuda.synchronize(dev)
    zt.grad = None
    wt.grad = None
    a, b, c = (torch.cuda.Event(enable_timing=True) for _ in range(3))
    a.record()
    out = W.demean(zt, eff, weights=wt, options=opts, solver=solver)
    loss = (vt * out).sum()
    b.record()
    loss.backward()
    c.record()
    torch.cuda.synchronize(dev)
    gw = wt.grad.cpu().numpy()
    gz = zt.grad.cpu().numpy()
    rng = np.random.default_rng(5)
    idx = rng.choice(z.size, 64, replace=False)
    h = 1e-6
    t_fd = time.perf_counter()

    def r_of(wv, zv):
        return W.Solver(eff, weights=wv, device=dev.index).solve(zv, opts).demeaned

    fd_w, fd_z = [], []
    base = solver.solve(z, opts).demeaned
    for i in idx:
        wp, wm = w.copy(), w.copy()
        wp[i] += h
        wm[i] -= h
        fd_w.append(float(v @ (r_of(wp, z) - r_of(wm, z))) / (2 * h))
        zp = z.copy()
        zp[i] += h
        fd_z.append(float(v @ (solver.solve(zp, opts).demeaned - base)) / h)
    fd_w, fd_z = np.array(fd_w), np.array(fd_z)
    t_fd = time.perf_counter() - t_fd
    return {"n": int(z.size), "forward_ms": a.elapsed_time(b), "backward_ms": b.elapsed_time(c),
            "grad_w_rel_err_vs_fd": float(np.max(np.abs(gw[idx] - fd_w)) / np.max(np.abs(fd_w))),
            "grad_z_rel_err_vs_fd": float(np.max(np.abs(gz[idx] - fd_z)) / np.max(np.abs(fd_z))),
            "fd_s": t_fd,
            "fd": "central differences, step 1e-6, 64 random weight coordinates (new Solver per "
                  "perturbation); forward differences for the same 64 z coordinates (linear); tol 1e-13"}


def run_ours(args):
    import torch
    rank, world, local = dist_env()
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600))
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)
    import within_b200 as W
    from within_b200 import _ffi
    # the reference's published configuration first, in a process not yet holding the 10M-row
    # workload (its wall clock covers host work: set-up is mostly host code)
    published = None if (args.no_published or world > 1) else published_section(W, args)
    codes, y = workload(args.rows)
    t0 = time.perf_counter()
    solver = W.Solver(codes, device=local, tuning=tuning_arg(args))
    t_setup = time.perf_counter() - t0
    n, nd = solver.n_obs, solver.n_dofs
    opts = W.LsmrOptions(tol=args.tol)
    yd = torch.tensor(y, device=dev)
    X = torch.empty((1, nd), dtype=torch.float64, device=dev).t()
    D = torch.empty((1, n), dtype=torch.float64, device=dev).t()
    stream = torch.cuda.current_stream(dev)
    for _ in range(args.warmup):
        solver.solve_device(yd, opts, X, D)
    torch.cuda.synchronize(dev)
    if world > 1:
        torch.distributed.barrier()
    L = _ffi.lib()
    L.within_launch_count_reset()
    with Clocks(local) as clk:
        torch.cuda.synchronize(dev)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        iters = []
        for _ in range(args.steps):
            _, _, st = solver.solve_device(yd, opts, X, D)
            iters.append(st[0][1])
        e1.record(stream)
        torch.cuda.synchronize(dev)
    launches = int(L.within_launch_count())
    t_dev = e0.elapsed_time(e1) / 1e3
    if world > 1:
        torch.distributed.barrier()
    t_max = max_over_ranks(t_dev, world, dev)
    value = world * args.steps / t_max
    ms = t_max / args.steps * 1e3
    it = int(np.median(iters))
    # accuracy against the FP64 oracle solve at tol 1e-12 (plain GPU, same design)
    dm = D[:, 0].clone()
    Xr, Dr, st_ref = solver.solve_device(yd, W.LsmrOptions(tol=1e-12, maxiter=5000))
    err = demeaned_err(dm, Dr[:, 0], yd)
    # batched: k = 8 right-hand sides per solve_batch (one multi-RHS LSMR that
    # reads the design once per apply for all columns); solves/s = 8 / time
    from within_b200 import workloads as WL
    kb = 8
    Yb = torch.tensor(np.asfortranarray(WL.akm_response(n, kb, seed=13)), device=dev)
    Yb = Yb.t().contiguous().t()
    Xb = torch.empty((kb, nd), dtype=torch.float64, device=dev).t()
    Db = torch.empty((kb, n), dtype=torch.float64, device=dev).t()
    for _ in range(2):
        solver.solve_device(Yb, opts, Xb, Db)
    torch.cuda.synchronize(dev)
    b0, b1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    b0.record(stream)
    reps_b = max(1, args.steps // 2)
    for _ in range(reps_b):
        _, _, stb = solver.solve_device(Yb, opts, Xb, Db)
    b1.record(stream)
    torch.cuda.synchronize(dev)
    t_b = b0.elapsed_time(b1) / 1e3 / reps_b
    _, Dref_b, _ = solver.solve_device(Yb, W.LsmrOptions(tol=1e-12, maxiter=5000))
    err_b = demeaned_err(Db, Dref_b, Yb)
    batched = {"k": kb, "value": kb / t_b, "unit": UNIT, "ms_per_batch": t_b * 1e3,
               "iterations_max": max(s_[1] for s_ in stb), "demeaned_err_vs_fp64_tol1e-12": err_b,
               "speedup_vs_single": (kb / t_b) / value * world}
    mixed = None if args.no_mixed else mixed_section(W, codes, dev, stream, args)
    many = None if (args.no_many or world > 1) else many_section(W, args)
    autograd = None if (args.no_autograd or world > 1) else autograd_section(W, dev)
    # e2e through the host API: y from page-locked host memory in, demeaned and
    # x out to page-locked host buffers, every step (Solver.solve)
    y_pin = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
    y_pin[:] = y
    x_pin = torch.empty(nd, dtype=torch.float64, pin_memory=True).numpy()
    d_pin = torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()
    for _ in range(2):
        solver.solve(y_pin, opts, x_out=x_pin, demeaned_out=d_pin)
    if world > 1:
        torch.distributed.barrier()
    t1 = time.perf_counter()
    for _ in range(args.steps):
        solver.solve(y_pin, opts, x_out=x_pin, demeaned_out=d_pin)
    t_e2e = time.perf_counter() - t1
    t_e2e = max_over_ranks(t_e2e, world, dev)
    e2e = world * args.steps / t_e2e
    # the same with pageable numpy buffers (staged in chunks by the library)
    solver.solve(y, opts)
    t1 = time.perf_counter()
    reps_pg = max(2, args.steps // 2)
    for _ in range(reps_pg):
        solver.solve(y, opts)
    e2e_pageable = reps_pg / (time.perf_counter() - t1)
    # roofline: the operator pair A v / A^T u (the design operator) timed alone
    v = torch.randn(nd, dtype=torch.float64, device=dev)
    u = torch.randn(n, dtype=torch.float64, device=dev)
    av = torch.empty(n, dtype=torch.float64, device=dev)
    atu = torch.empty(nd, dtype=torch.float64, device=dev)
    s_ptr = stream.cuda_stream
    for _ in range(3):
        solver.operator_apply_device(v, av, s_ptr)
        solver.operator_apply_adjoint_device(u, atu, s_ptr)
    reps = 20
    ga, gb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    sa, sb = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ga.record(stream)
    for _ in range(reps):
        solver.operator_apply_device(v, av, s_ptr)
    gb.record(stream)
    sa.record(stream)
    for _ in range(reps):
        solver.operator_apply_adjoint_device(u, atu, s_ptr)
    sb.record(stream)
    torch.cuda.synchronize(dev)
    t_gather = ga.elapsed_time(gb) / 1e3 / reps
    t_scatter = sa.elapsed_time(sb) / 1e3 / reps
    Q = codes.shape[1]
    bytes_gather = 4 * Q * n + 8 * nd + 8 * n          # codes, x, y out
    bytes_scatter = 4 * Q * n + 8 * n + 8 * nd         # codes/permutation, u, out
    achieved = (bytes_gather + bytes_scatter) / (t_gather + t_scatter) / 1e9
    peak, peak_kind = peaks()
    traffic, traffic_src = pair_traffic(n, Q, solver)
    pc = solver.preconditioner
    ps = pc.stats() if pc is not None else None
    ib = iteration_bytes(n, nd, Q, k=1, ps=ps)
    t_solve = ms / 1e3
    whole = {"bytes_per_iteration": ib, "iterations": it, "preconditioner": ps,
             "gbs_survey": (ib["op_survey"] + ib["precond"] + ib["vectors"]) * it / t_solve / 1e9,
             "gbs_fused": (ib["op_fused"] + ib["precond"] + ib["vectors"]) * it / t_solve / 1e9,
             "note": "(B_op + B_M + B_vec) x iterations / device time of one solve (set-up and read-back "
                     "kernels included in the time, not in the bytes)"}
    whole["frac_survey"] = whole["gbs_survey"] / peaks()[0]
    whole["frac_fused"] = whole["gbs_fused"] / peaks()[0]
    roof = {"bound": "hbm",
            "kernel": "design operator pair: within_solver_operator_apply (D v) + "
                      "within_solver_operator_apply_adjoint (D^T u), the kernels the solver selects for the design",
            "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
            "peak_kind": peak_kind, "traffic": traffic, "traffic_source": traffic_src,
            "gather_gbs": bytes_gather / t_gather / 1e9, "scatter_gbs": bytes_scatter / t_scatter / 1e9,
            "algorithmic_bytes_per_launch": {"gather": bytes_gather, "scatter": bytes_scatter}}
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic", "config": config_dict(n, nd),
        "iterations": it, "lsmr_iters_per_s": world * sum(iters) / t_max, "setup_s": t_setup,
        "demeaned_err_vs_fp64_tol1e-12": err, "whole_solve": whole, "batched_fp64": batched,
        "mixed_batched": mixed,
        "many_designs": many, "autograd": autograd, "published_config": published,
        "roofline": roof,
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": 8 * n,
                "d2h_bytes_per_step": 8 * (n + nd),
                "path": "Solver.solve, page-locked numpy y in, demeaned and x out (host clock)",
                "pageable_numpy_value": e2e_pageable},
        "gpu_launches": launches, "clocks": clk.summary(),
    }
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            s, t_cs, t_it = cpu_baseline(codes, y, args.tol, args.cpu_sample_iters)
            cpu_solve = t_it * it
            line["cpu_baseline"] = {
                "value": 1.0 / cpu_solve, "unit": UNIT, "cores": os.cpu_count() or 1, "kind": "port",
                "sample": f"{args.cpu_sample_iters} LSMR iterations of the C++ restatement on the same "
                          f"design ({t_it * 1e3:.0f} ms/iteration on {os.cpu_count() or 1} host threads), "
                          f"scaled to the GPU "
                          f"solve's {it} iterations; its setup {t_cs:.1f}s excluded"}
        except Exception as e:  # the baseline must not sink the GPU line
            line["cpu_baseline"] = {"value": None, "unit": UNIT, "cores": os.cpu_count() or 1, "kind": "port",
                                    "sample": f"failed: {e}"}
    if rank == 0:
        print(json.dumps(line), flush=True)
    del solver
    if world > 1:
        torch.distributed.barrier()
        torch.distributed.destroy_process_group()


def _run_counts(codes):
    """Runs (maximal stretches of equal codes) per term along the design's
    internal order: the worker-sorted panel is already in that order."""
    c = np.asarray(codes)
    return [int(1 + np.count_nonzero(c[1:, t] != c[:-1, t])) for t in range(c.shape[1])]


def kernel_byte_model(n, nd, Q, ps, runs, weighted=False, s=8):
    """Algorithmic bytes per LSMR iteration of each kernel family of the FP64
    one-column solve (codes 4 B, values s B; every index and value read once,
    every result written once):
      row sweep (LSMR step)  4nQ + 2sn (u read, write) + s nd (coefficients
                             gathered once) + s nd (A^T u / run sums out)
      row sweep (adjoint)    4nQ + sn + s nd;  gather / demean: 4nQ + sn (+ sn y) + s nd
      run combine            the run sums and their level-sorted order (4 + s per run) + s per level
      C^T, C, factor rounds, dense blocks, core: (4 + 2s) per non-zero + 2s per row
      restrict (4 + 3s), means 2s, prolongation (4 + s) per local slot, + s nd out
      p~ 3s nd, alpha step 2s nd, solution update 7s nd;  set-up kernels per solve.
    Returns {family: (bytes per iteration, launches of the family per iteration)}."""
    w = s * n if weighted else 0
    slots = ps.get("n_slots", 0) if ps else 0
    red = ps.get("n_reduced", 0) if ps else 0
    combine = sum(r for r, t in zip(runs, range(Q)) if 0 < r < n // 3) * (4 + s)
    m = {
        "sweep_lsmr": 4 * n * Q + 2 * s * n + 2 * s * nd + w,
        "sweep_adjoint": 4 * n * Q + s * n + s * nd + w,
        "gather": 4 * n * Q + s * n + s * nd + w,
        "demean": 4 * n * Q + 2 * s * n + s * nd,
        "ScatterF": combine + s * nd,
        "ptilde": 3 * s * nd, "alpha": 2 * s * nd, "solution_update": 7 * s * nd,
    }
    if ps and ps.get("n_subdomains"):
        m.update({
            "CtF": ps["nnz_ct"] * (4 + 2 * s) + 2 * s * red,
            "CF": ps["nnz_c"] * (4 + 2 * s) + 2 * s * (slots - red),
            "FwdF": ps["nnz_fwd"] * (4 + 2 * s) + 2 * s * red,
            "BwdF": ps["nnz_bwd"] * (4 + 2 * s) + 2 * s * red,
            "DenseF": ps["nnz_dense"] * (4 + 2 * s),
            "CoreF": ps["nnz_core"] * (4 + 2 * s),
            "RestrictF": slots * (4 + 3 * s),
            "MeanF": slots * 2 * s,
            "KeptSumF": 2 * s * red,
            "ProlongF": slots * (4 + s) + s * nd,
        })
    return m


def _family(name):
    import re
    if name.startswith("k_tsweep") or name.startswith("k_rowsweep"):
        args = re.findall(r"<([^>]*)>", name)
        mode = args[0].split(",")[1].strip() if args else "1"
        return "sweep_lsmr" if mode == "1" else ("sweep_adjoint" if mode == "0" else None)
    if name.startswith("k_tgather"):
        return "demean" if name.rstrip(">").endswith("true") else "gather"
    if name.startswith("k_apply"):
        return "gather"
    if name.startswith("k_demean"):
        return "demean"
    if name.startswith("k_csweep"):
        mode = name.split(",")[1].strip()
        return "sweep_lsmr" if mode == "1" else ("sweep_adjoint" if mode == "0" else None)
    if name.startswith("k_rounds"):   # all narrow rounds of one direction
        return "BwdF" if name.rstrip(">").rstrip().endswith("true") else "FwdF"
    for f in ("ScatterF", "CtF", "CF<", "FwdF", "BwdF", "DenseF", "CoreF", "RestrictF", "MeanF", "KeptSumF",
              "ProlongF"):
        # the list engine's functors are named Sl<step><K>, the others' <step>F<K, type>
        if f in name or "Sl" + f.rstrip("<")[:-1] + "<" in name:
            return f.rstrip("<")
    for k, f in (("k_ptilde", "ptilde"), ("k_alpha_step", "alpha"), ("k_solution_update", "solution_update")):
        if name.startswith(k):
            return f
    return None


def kernel_timeline(args):
    """Per-kernel device durations of one solve of the bench workload, from
    CUPTI timestamps (torch.profiler), with the loop replayed as two-iteration
    graphs (WITHIN_GRAPH_LOOP=0) so that every iteration's launches are
    recorded, in plain stream order (WITHIN_PDL=0).  For each kernel: launches, mean and total device time; for
    each kernel family of the FP64 solve, its algorithmic bytes per
    iteration (kernel_byte_model), its device time per iteration and the
    achieved GB/s and fraction of the HBM peak."""
    import collections
    import re
    os.environ["WITHIN_GRAPH_LOOP"] = "0"
    # plain stream order: with programmatic dependent launch a kernel starts
    # early and waits in-kernel, so its recorded span would include its
    # predecessor's tail
    os.environ["WITHIN_PDL"] = "0"
    import torch
    from torch.profiler import ProfilerActivity, profile
    import within_b200 as W
    codes, y = workload(args.rows)
    dev = torch.device("cuda", 0)
    if args.kernel_timeline == "mixed":
        rng = np.random.default_rng(4)
        w = rng.lognormal(0.0, 1.0, codes.shape[0])
        s = W.Solver(codes, weights=w, precision="mixed", tuning=tuning_arg(args))
        Y = torch.tensor(np.asfortranarray(rng.standard_normal((codes.shape[0], 4))), device=dev)
        Y = Y.t().contiguous().t()
    else:
        s = W.Solver(codes, tuning=tuning_arg(args))
        Y = torch.tensor(y, device=dev)
    opts = W.LsmrOptions(tol=args.tol)
    for _ in range(2):
        _, _, st = s.solve_device(Y, opts)
    iters = st[0][1]
    torch.cuda.synchronize(dev)
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        s.solve_device(Y, opts)
        torch.cuda.synchronize(dev)
    dur = collections.defaultdict(list)
    for e in prof.events():
        if e.device_type == torch.autograd.DeviceType.CUDA and (e.name.startswith("void wgpu::") or
                                                                  e.name.startswith("wgpu::")):
            nm = re.sub(r"\(.*", "", e.name).replace("void ", "").replace("wgpu::", "")
            dur[nm].append(e.device_time_total if hasattr(e, "device_time_total") else e.cuda_time_total)
    out = {k: {"launches": len(v), "mean_us": float(np.mean(v)), "median_us": float(np.median(v)),
               "total_us": float(np.sum(v))}
           for k, v in sorted(dur.items(), key=lambda kv: -sum(kv[1]))}
    fam = None
    if args.kernel_timeline == "fp64":
        pc = s.preconditioner
        ps = pc.stats() if pc is not None else None
        model = kernel_byte_model(codes.shape[0], s.n_dofs, codes.shape[1], ps, _run_counts(codes))
        peak = peaks()[0]
        tot = collections.defaultdict(float)
        for k, v in dur.items():
            f = _family(k)
            if f:
                tot[f] += float(np.sum(v))
        fam = {}
        for f, us in sorted(tot.items(), key=lambda kv: -kv[1]):
            per_it = us / max(1, iters) if f not in ("demean", "sweep_adjoint") else us
            b = model.get(f)
            gbs = b / (per_it * 1e-6) / 1e9 if b and per_it > 0 else None
            fam[f] = {"us_per_iteration": per_it, "bytes_per_iteration": b, "gbs": gbs,
                      "frac_of_peak": gbs / peak if gbs else None}
        fam["_note"] = ("demean and the adjoint sweep run once per solve (their time is the launch, not per "
                        "iteration); iterations = %d; peak %.1f GB/s (%s)" % (iters, peak, peaks()[1]))
    print(json.dumps({"kernel_timeline": args.kernel_timeline, "rows": args.rows, "iterations": iters,
                      "kernels": out, "families": fam}, indent=1))


_SETUP_CHILD = r"""
import json, sys, time
import numpy as np
import within_b200 as W
from within_b200 import workloads as WL
wl = sys.argv[1]
if wl == "akm10m":
    codes = WL.akm_panel(); y = np.random.default_rng(7).standard_normal(codes.shape[0]); tol = 1e-8
else:
    codes, y = WL.fixest_like(); tol = 1e-6
opts = W.LsmrOptions(tol=tol, maxiter=200)
best = None
for rep in range(3):
    print("=== rep", rep, file=sys.stderr, flush=True)
    t0 = time.perf_counter(); s = W.Solver(codes); t1 = time.perf_counter()
    r = s.solve(y, opts); t2 = time.perf_counter()
    cur = (t2 - t0, t1 - t0, t2 - t1, int(r.iterations), rep)
    best = cur if best is None or cur[0] < best[0] else best
    del s
print(json.dumps({"workload": wl, "best_total_ms": best[0] * 1e3, "new_ms": best[1] * 1e3,
                  "first_solve_ms": best[2] * 1e3, "iterations": best[3], "best_rep": best[4]}))
"""


def setup_trace(args):
    """Solver::new + first solve of two designs with the set-up's phase trace."""
    env = dict(os.environ)
    env["WITHIN_TRACE"] = "1"
    root = os.path.dirname(os.path.abspath(__file__))
    env["PYTHONPATH"] = root + os.pathsep + env.get("PYTHONPATH", "")
    for wl in ("fixest", "akm10m"):
        out = subprocess.run([sys.executable, "-c", _SETUP_CHILD, wl], capture_output=True, text=True,
                             timeout=900, env=env)
        if out.returncode:
            print(out.stderr[-3000:], flush=True)
            raise SystemExit(out.returncode)
        res = json.loads(out.stdout.strip().splitlines()[-1])
        reps = out.stderr.split("=== rep ")
        trace = reps[res["best_rep"] + 1] if len(reps) > res["best_rep"] + 1 else ""
        print(json.dumps(res), flush=True)
        print("\n".join(l for l in trace.splitlines() if "within trace" in l), flush=True)


def main():
    args = parse()
    if args.setup_trace:
        setup_trace(args)
        return
    if args.kernel_timeline:
        kernel_timeline(args)
        return
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
