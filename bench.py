#!/usr/bin/env python
"""Benchmark of the Tapas N-body evaluation path on B200.

Workload (one step = one full FMM evaluation: octree build, upward pass,
dual-tree traversal with M2L + P2P, downward pass):
  N = 16,000,000 bodies uniform on the unit sphere surface, charges U[-1,1]
  minus their mean, requested relative-L2 potential error 1e-6.  Parameters
  (P, theta, ncrit) come from the learned chooser: its shortlist (the fastest
  candidates predicted to come within 0.25 in log10 of the tolerance, then the
  margin-safe choice) is verified against an FP64 direct sum on 4,000 sampled
  targets and the ones that meet it are run twice more, timed (all before the
  timed region); the fastest of them is timed, the rule table's setting if
  none meets it.

Printed JSON line (rank 0):
  value       particles/s of the mixed form, inputs resident in HBM
  e2e         the same through the C-ABI evaluate() call with pinned HOST
              buffers: host->device copy of the bodies and device->host copy of
              the results inside the timed region
  fp64        the plain FP64 form (same chooser tolerance rule) for reference
  roofline    the dominant kernel of the step against its bound
  cpu_baseline  the reference's own CPU implementation (oracle/_ref, built from
              the reference sources) on a bounded sample of the same workload
  configs     the other measured configurations: 100k cube against the
              reference's own output, 1M Plummer (FP64 vs mixed), 4M-body
              Barnes-Hut (skipped with --no-configs)

Multi-GPU: replicas only (the path is one tree per GPU); each rank evaluates its
own seeded body set, value = all ranks' bodies / max-over-ranks time.
``--impl reference`` times the reference CPU implementation instead.
"""
from __future__ import annotations

import argparse
import importlib.util
import json
import os
import pathlib
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = pathlib.Path(__file__).resolve().parent
METRIC = "FMM particles/s at 1e-6 rel-L2: mixed+learned vs plain FP64 on 1 B200"
WORKLOAD = "sphere_surface"


def load_package():
    if "tapas_reduce_b200" in sys.modules:
        return sys.modules["tapas_reduce_b200"]
    pkg_dir = ROOT / "tapas-reduce_b200"
    spec = importlib.util.spec_from_file_location(
        "tapas_reduce_b200", pkg_dir / "__init__.py", submodule_search_locations=[str(pkg_dir)])
    mod = importlib.util.module_from_spec(spec)
    sys.modules["tapas_reduce_b200"] = mod
    spec.loader.exec_module(mod)
    return mod


def load_oracle():
    sys.path.insert(0, str(ROOT / "oracle"))
    import oracle
    return oracle


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index: int):
        self.dev = device_index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.dev}", f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
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
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": []}
        if not self.path or not os.path.exists(self.path):
            return out
        rows = []
        for line in open(self.path):
            parts = [p.strip() for p in line.split(",")]
            if len(parts) >= 9:
                rows.append(parts)
        if not rows:
            return out
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in rows:
            for i, nme in enumerate(names):
                if r[5 + i].lower().startswith("active"):
                    reasons.add(nme)
        out["sm_mhz"] = float(np.median(sm)) if sm else None
        out["sm_max_mhz"] = max(mx) if mx else None
        out["reasons"] = sorted(reasons)
        out["samples"] = len(rows)
        os.unlink(self.path)
        return out


# ---------------------------------------------------------------------------
# distributed plumbing (replicas)
# ---------------------------------------------------------------------------
def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    pg = None
    if world > 1:
        import datetime
        import torch.distributed as tdist
        tdist.init_process_group("gloo", timeout=datetime.timedelta(seconds=600))
        pg = tdist
    return world, rank, local, pg


def barrier(pg):
    if pg is not None:
        pg.barrier()


def max_over_ranks(pg, v: float) -> float:
    if pg is None:
        return v
    import torch
    t = torch.tensor([v], dtype=torch.float64)
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    return float(t.item())


def sum_over_ranks(pg, v: float) -> float:
    if pg is None:
        return v
    import torch
    t = torch.tensor([v], dtype=torch.float64)
    pg.all_reduce(t, op=pg.ReduceOp.SUM)
    return float(t.item())


def replica_throughput(pg, ms: float, n: int):
    """Whole-job throughput of independent replicas: every rank's bodies over
    the slowest rank's step time.  Returns (max ms, total bodies, bodies/s)."""
    ms_max = max_over_ranks(pg, ms)
    n_total = sum_over_ranks(pg, float(n))
    return ms_max, n_total, n_total / (ms_max * 1e-3)


# ---------------------------------------------------------------------------
# reference CPU implementation (oracle/_ref, built from the reference sources)
# ---------------------------------------------------------------------------
REF_SAMPLE_N = 50_000
# The setting the reference runs on its samples: the one the learned chooser
# picks for the 16M sphere-surface workload (and one of the sampled reference
# outputs of that workload was made with), so both arms evaluate the same
# method.
REF_P, REF_THETA, REF_NCRIT = 12, 0.35, 128
GOLDEN = ROOT / "tests" / "golden"


def cpu_reference_run(tb, orc, n=REF_SAMPLE_N, seed=77):
    """One evaluation of the reference FMM on a bounded sample of the
    workload (same distribution, n bodies) on one host core; particles/s."""
    x, y, z, q = tb.datasets.make(WORKLOAD, n, seed)
    if orc.reference_available(REF_P):
        r = orc.run_reference(x, y, z, q, P=REF_P, ncrit=REF_NCRIT, theta=REF_THETA)
        t = r["times"]
        secs = t["tree"] + t["upward"] + t["traverse"] + t["downward"]
        kind = "reference"
    else:
        t0 = time.perf_counter()
        orc.Oracle(x, y, z, q, P=REF_P, ncrit=REF_NCRIT, theta=REF_THETA)
        secs = time.perf_counter() - t0
        kind = "port"
    return n / secs, kind, secs


def host_threads() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def cpu_reference_parallel(tb, orc, n, seed, workers):
    """``workers`` concurrent reference runs, one per host thread, each on its
    own bounded sample (seeds seed..seed+workers-1).  The reference build here
    has neither a threading backend nor MPI, so independent processes are how
    it uses every host thread; the aggregate (all bodies over the slowest run)
    is the throughput of perfectly scaled replicas."""
    from concurrent.futures import ThreadPoolExecutor
    if workers <= 1:
        v, kind, secs = cpu_reference_run(tb, orc, n=n, seed=seed)
        return v, kind, secs
    with ThreadPoolExecutor(max_workers=workers) as ex:
        runs = list(ex.map(lambda k: cpu_reference_run(tb, orc, n=n, seed=seed + 7919 * k),
                           range(workers)))
    slowest = max(r[2] for r in runs)
    return workers * n / slowest, runs[0][1], slowest


def reference_scaling_evidence():
    """Per-particle rate of the reference (1 core, same distribution and
    setting) at the sizes its sampled outputs were made at: it shows how the
    bounded-sample rate carries to the full workload."""
    out = {}
    for name in ("refsample_sphere_n1000000_p15", "refsample_sphere_n16000000_p15",
                 "refsample_sphere_n16000000_p13", "refsample_sphere_n16000000_p12"):
        f = GOLDEN / f"{name}.npz"
        if f.exists():
            g = np.load(f)
            key = f"n{int(g['n'])}_P{int(g['P'])}_theta{float(g['theta']):g}"
            out[key] = _r(int(g["n"]) / float(g["ref_seconds"]))
    return out


def cpu_baseline_obj(value, kind, secs, n=REF_SAMPLE_N, cores=1):
    who = ("1 rank x 1 thread (the reference's Serial threading)" if cores == 1 else
           f"{cores} concurrent single-thread reference processes, one per host thread, "
           f"each on its own sample of {n} bodies")
    return {"value": value, "unit": "particles/s", "cores": cores, "kind": kind,
            "sample": f"{n} bodies of the same sphere-surface workload, "
                      f"P={REF_P} theta={REF_THETA} ncrit={REF_NCRIT} (the setting the "
                      f"chooser picks for this workload), "
                      f"{who}, {secs:.2f} s",
            "ref_rate_at_full_sizes_1core": reference_scaling_evidence()}


def run_reference_arm(args):
    world, rank, _, pg = dist_setup(args)
    if rank != 0:
        return 0
    tb = load_package()
    orc = load_oracle()
    vals = []
    kind = secs = None
    ns = args.ref_sample
    cores = args.ref_threads if args.ref_threads > 0 else min(host_threads(), 128)
    for i in range(args.warmup + args.steps):
        v, kind, secs = cpu_reference_parallel(tb, orc, ns, 77 + 100_003 * i, cores)
        if i >= args.warmup:
            vals.append(v)
    value = float(np.mean(vals))
    line = {"metric": METRIC, "value": value, "unit": "particles/s", "impl": "reference",
            "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": cores * ns / value * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"{WORKLOAD} samples, {cores} x n={ns} per step",
                       "P": REF_P, "theta": REF_THETA, "ncrit": REF_NCRIT,
                       "host_threads": cores},
            "cpu_baseline": cpu_baseline_obj(value, kind, secs, ns, cores),
            "e2e": {"value": value, "unit": "particles/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0},
            "gpu_launches": 0}
    print(json.dumps(line), flush=True)
    return 0


# ---------------------------------------------------------------------------
# our arm
# ---------------------------------------------------------------------------
def _r(v, sig=4):
    """A float rounded to `sig` significant digits (keeps the JSON line short)."""
    if v is None or isinstance(v, (bool, int, str)):
        return v
    v = float(v)
    if v == 0 or not np.isfinite(v):
        return v
    return float(f"{v:.{sig}g}")


def _rr(obj):
    if isinstance(obj, dict):
        return {k: _rr(v) for k, v in obj.items()}
    if isinstance(obj, (list, tuple)):
        return [_rr(v) for v in obj]
    return _r(obj) if isinstance(obj, float) else obj


def choose(tb, n, tol, precision):
    from importlib import import_module
    chooser = import_module("tapas_reduce_b200.chooser")
    return chooser.choose_params(n=n, tol=tol, precision=precision)


def reference_sample(name):
    """Sampled FP64 output of the unmodified reference on a seeded body set
    (tests/golden/refsample_*.npz): (indices, values, setting) or None."""
    f = GOLDEN / f"{name}.npz"
    if not f.exists():
        return None
    g = np.load(f)
    return g["idx"], g["trg"], (int(g["P"]), float(g["theta"]), int(g["ncrit"]))


def rel_l2_pair(a, b):
    ep = np.linalg.norm(a[:, 0] - b[:, 0]) / np.linalg.norm(b[:, 0])
    ea = np.linalg.norm(a[:, 1:] - b[:, 1:]) / np.linalg.norm(b[:, 1:])
    return float(ep), float(ea)


def verified(ctx, tb, orc, dev, out_dev, tries, d_check, tg, tol, precision, timer=None):
    """The setting of `tries` to time: each is run and checked against the FP64
    direct sum on the sampled targets; of those that meet `tol`, the fastest by
    `timer(setting)` (ms of one more evaluation; with no timer, the first).
    Returns (setting, the ones that missed)."""
    missed, met = [], []
    for cand in tries:
        cand = dict(cand)
        try:
            ctx.evaluate(*dev, P=cand["P"], ncrit=cand["ncrit"], theta=cand["theta"],
                         precision=precision, out=out_dev)
            e = orc.rel_l2(out_dev.cpu().numpy()[tg], d_check)[0]
        except tb.TapasError as err:  # e.g. a setting too large for device memory
            cand["error"] = str(err)
            e = float("inf")
        cand["verified_rel_l2_pot"] = e
        if e <= tol:
            if timer is None:
                return cand, missed
            cand["measured_ms"] = timer(cand)
            met.append(cand)
        else:
            missed.append(cand)
    if not met:
        return None, missed
    best = min(met, key=lambda c: c["measured_ms"])
    best["also_verified"] = [{k: _r(c[k]) for k in ("P", "theta", "ncrit", "measured_ms")}
                             for c in met if c is not best]
    return best, missed


def device_time(torch, stream, step, steps, warmup, pg, clocks=None):
    """CUDA-event milliseconds per step on `stream` (max over ranks), after
    `warmup` untimed steps, bracketed by barriers and synchronisations."""
    for _ in range(warmup):
        step()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier(pg)
    torch.cuda.synchronize()
    if clocks is not None:
        clocks.__enter__()
    try:
        ev0.record(stream)
        for _ in range(steps):
            step()
        ev1.record(stream)
        torch.cuda.synchronize()
    finally:
        if clocks is not None:
            clocks.__exit__(None, None, None)
    barrier(pg)
    return max_over_ranks(pg, ev0.elapsed_time(ev1) / steps)


def profiled_phases(ctx, step):
    """Phase times (ms) of one extra, untimed step with per-phase events."""
    ctx.set_profiling(True)
    try:
        step()
        return ctx.timings()
    finally:
        ctx.set_profiling(False)


def phases_compact(ph):
    keys = ("bbox_keys", "sort", "tree", "p2m", "m2m", "traverse", "list_sort", "m2l_setup",
            "m2l_tc", "m2l_fp64", "m2l", "p2p", "l2l", "l2p", "download")
    return {k: _r(ph.get(k, 0.0)) for k in keys if ph.get(k, 0.0) > 0}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=16_000_000)
    ap.add_argument("--tol", type=float, default=1e-6)
    ap.add_argument("--targets", type=int, default=4000)
    ap.add_argument("--P", type=int, default=0, help="with --theta and --ncrit: fixed setting "
                                                     "instead of the learned choice")
    ap.add_argument("--theta", type=float, default=0.0)
    ap.add_argument("--ncrit", type=int, default=0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--no-configs", action="store_true",
                    help="skip the other configurations (100k cube, 1M Plummer, 1M sphere, "
                         "4M Barnes-Hut)")
    ap.add_argument("--ref-sample", type=int, default=REF_SAMPLE_N,
                    help="bodies per reference CPU step (--impl reference)")
    ap.add_argument("--ref-threads", type=int, default=0,
                    help="concurrent reference processes (--impl reference; 0 = all host "
                         "threads, at most 128)")
    args = ap.parse_args()
    if args.impl == "reference":
        return run_reference_arm(args)

    import torch
    world, rank, local, pg = dist_setup(args)
    torch.cuda.set_device(local)
    tb = load_package()
    n = args.n
    seed = 5 + 1000 * rank
    x, y, z, q = tb.datasets.make(WORKLOAD, n, seed=seed)
    tg = tb.datasets.sample_targets(n, args.targets, seed=99 + rank)
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z, q)]
    pinned = [torch.from_numpy(a).pin_memory() for a in (x, y, z, q)]
    out_dev = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    out_pin = torch.empty((n, 4), dtype=torch.float64).pin_memory()
    ctx = tb.Context(local)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    orc = load_oracle()

    # Learned choice (features of the body set, one batched network pass),
    # verified against the FP64 direct sum before timing; on a miss the rule
    # table's setting is used instead.
    from importlib import import_module
    chooser = import_module("tapas_reduce_b200.chooser")
    feats = None
    if args.P and args.theta and args.ncrit:
        # fixed setting (profiling a given configuration); still verified
        tries = [{"P": args.P, "theta": args.theta, "ncrit": args.ncrit, "precision": "mixed",
                  "source": "fixed by --P/--theta/--ncrit"}]
        ctx.partition(*dev, ncrit=args.ncrit)  # the direct-sum check reads the bodies
    else:
        # the learned chooser's shortlist; each is verified against the direct
        # sum, and of those that meet tol the fastest (one timed run each) is used
        feats = chooser.system_features(ctx, *dev)
        tries = chooser.candidates(ctx, feats, n, args.tol, "mixed", k=6)

    def timer_for(precision):
        """This rank's device ms of an evaluation of a setting, the faster of
        two (no collective: ranks may verify different shortlists)."""
        def t(c):
            best = float("inf")
            for _ in range(2):
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                ctx.evaluate(*dev, P=c["P"], ncrit=c["ncrit"], theta=c["theta"],
                             precision=precision, out=out_dev)
                e1.record(stream)
                e1.synchronize()
                best = min(best, float(e0.elapsed_time(e1)))
            return best
        return t

    d_check = ctx.direct(tg)
    prm, missed = verified(ctx, tb, orc, dev, out_dev, tries, d_check, tg, args.tol, tb.MIXED,
                           timer=timer_for(tb.MIXED))
    if prm is None:  # no candidate verified: the rule table's setting
        prm = choose(tb, n, args.tol, "mixed")
    if missed:
        prm["missed_before"] = [{k: _r(v) for k, v in m.items() if k in
                                 ("P", "theta", "ncrit", "verified_rel_l2_pot")} for m in missed]
    P, theta, ncrit = prm["P"], prm["theta"], prm["ncrit"]
    torch.cuda.synchronize()

    def step_dev():
        ctx.evaluate(*dev, P=P, ncrit=ncrit, theta=theta, precision=tb.MIXED, out=out_dev)

    def step_e2e():
        ctx.evaluate(*pinned, P=P, ncrit=ncrit, theta=theta, precision=tb.MIXED, out=out_pin)

    # ---- timed region: device-resident inputs, CUDA events on our stream ----
    ctx.set_profiling(False)
    for _ in range(args.warmup):
        step_dev()
    ctx.kernel_launches(reset=True)
    clk = ClockSampler(local)
    ms_max = device_time(torch, stream, step_dev, args.steps, 0, pg, clocks=clk)
    launches = ctx.kernel_launches() // args.steps
    clocks = clk.summary()
    _, n_total, value = replica_throughput(pg, ms_max, n)
    phases = profiled_phases(ctx, step_dev)  # one extra step with phase events
    li = ctx.list_info()
    ti = ctx.tree_info()

    # ---- accuracy: FP64 direct sum on sampled targets, reference's output ----
    res = out_dev.cpu().numpy()
    err = orc.rel_l2(res[tg], d_check)
    accuracy = {"rel_l2_pot": _r(err[0]), "rel_l2_acc": _r(err[1]), "targets": int(len(tg)),
                "meets_tol": bool(err[0] <= args.tol)}
    ref16 = None
    if n == 16_000_000 and rank == 0:  # the reference's output at our setting if made, else P=15
        for name in ("refsample_sphere_n16000000_p12", "refsample_sphere_n16000000_p13",
                     "refsample_sphere_n16000000_p15"):
            ref16 = reference_sample(name)
            if ref16 is not None and ref16[2] == (P, theta, ncrit):
                break
    if ref16 is not None:
        # the reference's FP64 output on the same bodies, at its own setting
        # (P, theta, ncrit) = reference_setting; at another setting of ours the
        # difference holds both evaluations' truncation errors
        e = rel_l2_pair(res[ref16[0]], ref16[1])
        accuracy.update(rel_l2_pot_vs_reference=_r(e[0]), rel_l2_acc_vs_reference=_r(e[1]),
                        reference_samples=int(len(ref16[0])),
                        reference_setting=list(ref16[2]))

    # ---- e2e through the C-ABI call with pinned host buffers, K steps ----
    for _ in range(2):
        step_e2e()
    barrier(pg)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        step_e2e()
    torch.cuda.synchronize()
    e2e_s = max_over_ranks(pg, (time.perf_counter() - t0) / args.steps)
    e2e = {"value": _r(n_total / e2e_s), "unit": "particles/s",
           "h2d_bytes_per_step": 4 * 8 * n, "d2h_bytes_per_step": 4 * 8 * n}

    # ---- plain FP64 form: at the mixed arm's setting, and its own learned choice ----
    # (rank 0 alone, no collectives: ranks may choose different settings)
    fp64 = None
    if not args.no_fp64 and rank == 0:
        fp64 = {}
        settings = [("same_setting", {"P": P, "theta": theta, "ncrit": ncrit,
                                      "source": "the mixed arm's setting"})]
        if feats is not None:
            c64, missed64 = verified(ctx, tb, orc, dev, out_dev,
                                     chooser.candidates(ctx, feats, n, args.tol, "fp64", k=4),
                                     d_check, tg, args.tol, tb.FP64, timer=timer_for(tb.FP64))
            if c64 is not None:
                settings.append(("learned_fp64", c64))
        for key, s64 in settings:
            def step64(s64=s64):
                ctx.evaluate(*dev, P=s64["P"], ncrit=s64["ncrit"], theta=s64["theta"],
                             precision=tb.FP64, out=out_dev)
            ms64 = device_time(torch, stream, step64, 2, 1, None)
            e64 = orc.rel_l2(out_dev.cpu().numpy()[tg], d_check)
            ph64 = profiled_phases(ctx, step64)
            li64, ti64 = ctx.list_info(), ctx.tree_info()
            rl64 = roofline_obj(ph64, li64, ti64, s64["P"], tb, precision="fp64")
            fp64[key] = {"ms_per_step": _r(ms64), "value": _r(n_total / (ms64 * 1e-3)),
                         "P": s64["P"], "theta": s64["theta"], "ncrit": s64["ncrit"],
                         "rel_l2_pot": _r(e64[0]), "rel_l2_acc": _r(e64[1]),
                         "meets_tol": bool(e64[0] <= args.tol),
                         "phases_ms": phases_compact(ph64),
                         "roofline": {k: _r(v) for k, v in rl64.items()
                                      if k in ("kernel", "ms", "bound", "achieved", "peak",
                                               "unit", "frac")},
                         "work": {"n_m2l": li64["n_m2l"],
                                  "n_p2p_interactions": li64["n_p2p_interactions"]}}
        ok = [v["ms_per_step"] for v in fp64.values() if v["meets_tol"]]
        if ok:
            fp64["mixed_speedup_vs_fastest_fp64_meeting_tol"] = _r(min(ok) / ms_max)

    # ---- roofline of the dominant kernel ----
    roofline = roofline_obj(phases, li, ti, P, tb)

    cpu = None
    if rank == 0 and not args.no_cpu_baseline:
        v, kind, secs = cpu_reference_run(tb, orc)
        cpu = cpu_baseline_obj(v, kind, secs)

    configs = None
    if rank == 0 and not args.no_configs:
        configs = {}
        for key, fn in (("cube_1e5", config_cube_100k), ("plummer_1e6", config_plummer_1m),
                        ("sphere_1e6_p15", config_sphere_1m),
                        ("barnes_hut_plummer_4e6", config_bh_4m)):
            try:
                configs[key] = _rr(fn(tb, orc, ctx, torch, stream))
            except Exception as err:  # reported, never fatal to the headline line
                configs[key] = {"error": str(err)[:200]}
            torch.cuda.empty_cache()

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": "particles/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_max,
                "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f32+f64", "data": "synthetic",
                "config": {"workload": f"{WORKLOAD} N={n} q=U[-1,1]-mean tol={args.tol}",
                           "bodies_per_gpu": n, "P": P, "theta": theta, "ncrit": ncrit,
                           "chooser": {k: _rr(v) for k, v in prm.items()
                                       if k not in ("P", "theta", "ncrit")},
                           "precision": "mixed",
                           "l2_flush": "inputs larger than L2 (512 MB of bodies per step)",
                           "parallelism": f"replicas x{world}"},
                "accuracy": accuracy, "e2e": e2e, "fp64": fp64,
                "phases_ms": phases_compact(phases),
                "work": {"n_m2l": li["n_m2l"], "n_p2p_interactions": li["n_p2p_interactions"],
                         "n_cells": ti["n_cells"], "max_depth": ti["max_depth"]},
                "roofline": _rr(roofline), "cpu_baseline": cpu, "clocks": clocks,
                "configs": configs, "gpu_launches": launches}
        print(json.dumps(line), flush=True)
    ctx.close()
    if pg is not None:
        pg.destroy_process_group()
    return 0


# ---------------------------------------------------------------------------
# the other measured configurations (rank 0, one GPU)
# ---------------------------------------------------------------------------
def _timed(torch, stream, fn, reps=3):
    """Median CUDA-event time (ms) of fn() on `stream` after one warm-up call."""
    fn()
    ts = []
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fn()
        e1.record(stream)
        torch.cuda.synchronize()
        ts.append(e0.elapsed_time(e1))
    return float(np.median(ts))


def _rel(a, b):
    return float(np.sqrt(np.sum((a - b) ** 2) / np.sum(b ** 2)))


def _fmm_config(tb, ctx, torch, stream, dist, n, seed, P, ncrit, theta, ntarg, tseed, refname):
    """Both forms at one setting: CUDA-event time, rel-L2 against the FP64
    direct sum on sampled targets and against the reference's own FP64 output
    on its sampled bodies (tests/golden/refsample_*)."""
    x, y, z, q = tb.datasets.make(dist, n, seed)
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z, q)]
    out = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    tg = tb.datasets.sample_targets(n, ntarg, seed=tseed)
    ref = reference_sample(refname)
    res = {"workload": f"{dist} N={n} P={P} theta={theta} ncrit={ncrit}"}
    if ref is not None:
        gf = np.load(GOLDEN / f"{refname}.npz")
        res["reference_1core_s"] = float(gf["ref_seconds"])
    for prec, name in ((tb.FP64, "fp64"), (tb.MIXED, "mixed")):
        ms = _timed(torch, stream, lambda: ctx.evaluate(*dev, P=P, ncrit=ncrit, theta=theta,
                                                         precision=prec, out=out))
        r = out.cpu().numpy()
        d = ctx.direct(tg)
        e = {"ms": ms, "particles_per_s": n / (ms * 1e-3),
             "rel_l2_pot_vs_direct": _rel(r[tg, 0], d[:, 0]),
             "rel_l2_acc_vs_direct": _rel(r[tg, 1:], d[:, 1:])}
        if ref is not None and ref[2] == (P, theta, ncrit):
            ep, ea = rel_l2_pair(r[ref[0]], ref[1])
            e["rel_l2_pot_vs_reference"] = ep
            e["rel_l2_acc_vs_reference"] = ea
        res[name] = e
    res["mixed_speedup"] = res["fp64"]["ms"] / res["mixed"]["ms"]
    return res


def config_cube_100k(tb, orc, ctx, torch, stream):
    """100,000 bodies uniform in [-1,1]^3, charges U[0,1] summing to 1, P=10,
    theta=0.4, ncrit=64 (the reference's CPU-runnable configuration)."""
    return _fmm_config(tb, ctx, torch, stream, "uniform_cube", 100_000, 101, 10, 64, 0.4, 1000,
                       7, "refsample_cube_n100000_p10")


def config_plummer_1m(tb, orc, ctx, torch, stream):
    """1M Plummer bodies (scale radius 1, r < 100), charges 1/N, P=10,
    theta=0.4, ncrit=64: plain FP64 against the mixed form."""
    return _fmm_config(tb, ctx, torch, stream, "plummer", 1_000_000, 102, 10, 64, 0.4, 2000, 8,
                       "refsample_plummer_n1000000_p10")


def config_sphere_1m(tb, orc, ctx, torch, stream):
    """1M sphere-surface bodies (the headline's distribution), zero-mean
    charges, at the headline's setting P=15, theta=0.4, ncrit=128."""
    return _fmm_config(tb, ctx, torch, stream, "sphere_surface", 1_000_000, 104, 15, 128, 0.4,
                       4000, 10, "refsample_sphere_n1000000_p15")


def config_bh_4m(tb, orc, ctx, torch, stream):
    """Barnes-Hut: 4M Plummer bodies, monopoles, theta=0.5, ncrit=32, softening
    1e-6: the FP32 walk (FP64 moments) and the FP64 walk; force error against
    a softened FP64 direct sum on 2,000 targets (self term included, as in the
    sample); interactions/s of the walk and tree-build bytes/s."""
    n = 4_000_000
    x, y, z, m = tb.datasets.make("plummer", n, 103)
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z, m)]
    out = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    tg = tb.datasets.sample_targets(n, 2000, seed=9)
    eps2 = 1e-6
    # softened FP64 direct sum for the sampled targets, on the GPU in chunks
    X = torch.stack(dev[:3], 1)
    M = dev[3]
    d = torch.zeros((len(tg), 4), dtype=torch.float64, device="cuda")
    tt = X[torch.from_numpy(tg).cuda()]
    chunk = 1 << 14  # 2,000 x 16,384 x 3 doubles = 0.8 GB per temporary
    for c0 in range(0, n, chunk):
        dx = X[None, c0:c0 + chunk, :] - tt[:, None, :]
        ir = torch.rsqrt((dx * dx).sum(-1) + eps2)
        mi = M[None, c0:c0 + chunk] * ir
        d[:, :3] += (dx * (mi * ir * ir)[..., None]).sum(1)
        d[:, 3] += mi.sum(1)
        del dx, ir, mi
    d = d.cpu().numpy()
    res = {"workload": "Barnes-Hut Plummer N=4e6 theta=0.5 ncrit=32 eps2=1e-6"}
    for prec, name in ((tb.MIXED, "fp32_walk"), (tb.FP64, "fp64_walk")):
        ctx.set_profiling(True)
        ms = _timed(torch, stream, lambda: ctx.bh_evaluate(*dev, ncrit=32, theta=0.5, eps2=eps2,
                                                            precision=prec, out=out))
        t = ctx.timings()
        ctx.set_profiling(False)
        na, nd = ctx.bh_counts()
        r = out.cpu().numpy()
        build_ms = t["bbox_keys"] + t["sort"] + t["tree"]
        res[name] = {"ms": ms, "interactions_per_s": (na + nd) / (ms * 1e-3),
                     "approx": na, "direct": nd,
                     "tree_build_ms": build_ms,
                     "tree_build_gbs": 244.0 * n / (build_ms * 1e-3) / 1e9,
                     "rel_l2_force_vs_direct": _rel(r[tg, :3], d[:, :3]),
                     "rel_l2_pot_vs_direct": _rel(r[tg, 3], d[:, 3])}
    return res


def _peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        return json.loads(p.read_text()), "measured"
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "sm_max_mhz": 1965.0}, "fallback"


def roofline_obj(phases, li, ti, P, tb, precision="mixed"):
    """Dominant kernel of the step and its roofline."""
    peaks, src = _peaks()
    from importlib import import_module
    rl = import_module("tapas_reduce_b200.roofline")
    return rl.dominant(phases, li, ti, P, peaks, src, precision=precision)


if __name__ == "__main__":
    sys.exit(main())
