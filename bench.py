#!/usr/bin/env python3
"""Throughput benchmark: decomposed nodes/s of the IVM branch-and-bound on the
50-job x 20-machine instance (U[1,99], seed 2), weak bound refined by the
Johnson two-machine bound (boundingMode 2), MinMin branching, initial upper
bound from NEH, 65536 explorers.

A step is one exploration window of `--window` seconds of device time on the
resident search (the tree is far too large to finish; the search continues
across steps).  `value` = decomposed nodes in the K timed steps / their
CUDA-event time, summed over ranks, time = max over ranks.  `e2e` is the same
metric through the C ABI from host memory: engine creation (instance upload
and table build), root + unfold, one window, result read-back, destroy.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--window S] [--impl reference]

Under torchrun each rank explores its own slice of the permutation space
(factoradic sub-interval of the root level); between windows the ranks
exchange the best makespan (a 4-byte MIN all-reduce) and an idle rank takes
half of the busiest rank's intervals (pbbperm_b200.distributed.rebalance).
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

N_JOBS, N_MACH, SEED = 50, 20, 2
NB_IVMS = 65536
# explorer-kernel DRAM traffic (read + write) per second of window, from
# `ncu --set full` on this workload (dram__bytes_read.sum + dram__bytes_write.sum
# = 117.4 MB + 1.864 GB over a 50.1 ms launch: the pair bounds stored by level)
NCU_DRAM_BYTES_PER_S = (117.418752e6 + 1.863688e9) / 0.050086912
BOUND_MODE, BRANCH_MODE = 2, 3
METRIC = "decomposed nodes/s (50x20, Johnson LB)"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--window", type=float, default=6.0)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=2)
    ap.add_argument("--cpu-sample", type=float, default=15.0)
    ap.add_argument("--workload", default="nodes", choices=["nodes", "batch", "serve"],
                    help="nodes: 50x20 nodes/s (default); batch: 512 uneven instances in one pool vs one at a "
                         "time; serve: Poisson request stream through the pool vs each request alone")
    ap.add_argument("--batch-count", type=int, default=512)
    ap.add_argument("--rates", default="10,100,500,2000")
    ap.add_argument("--serve-seconds", type=float, default=20.0, help="serve: stream length at each rate")
    ap.add_argument("--serve-requests", type=int, default=20000, help="serve: requests per rate at most")
    ap.add_argument("--solo-sample", type=int, default=200,
                    help="serve: requests timed through the single-instance engine")
    ap.add_argument("--batch-solo", type=int, default=0, help="batch: instances solved one at a time (0: all)")
    ap.add_argument("--warps-per-cta", type=int, default=0, help="explorer warps per CTA (0: as many as fit)")
    ap.add_argument("--pool-window", type=float, default=0.0,
                    help="device time per pool window (batch; 0: the autotuner's choice)")
    ap.add_argument("--config2", type=int, default=1, help="add the 20x20 solve-to-completion sub-object (N=1)")
    ap.add_argument("--mode1", type=int, default=1,
                    help="add the 50x20 Johnson-only (boundingMode 1) sub-object (N=1)")
    ap.add_argument("--summary-batch", type=int, default=128,
                    help="add a compact batched sub-object over this many instances (0: none; N=1)")
    ap.add_argument("--summary-serve", type=int, default=200,
                    help="add a compact served sub-object over this many requests (0: none; N=1)")
    ap.add_argument("--summary-rate", type=float, default=1000.0, help="request rate of the served sub-object")
    return ap.parse_args()


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def workload_config(extra=None):
    cfg = {"workload": "pfsp-50x20-u1-99-seed2", "n_jobs": N_JOBS, "n_machines": N_MACH, "seed": SEED,
           "bounding_mode": BOUND_MODE, "branching_mode": BRANCH_MODE, "nb_ivms": NB_IVMS,
           "initial_ub": "NEH", "l2": "explorer state (65536 x 22.7 KB) exceeds L2; no flush"}
    if extra:
        cfg.update(extra)
    return cfg


# ---------------------------------------------------------------------------
# CPU baseline: the reference multicore B&B (oracle/_ref/bbJ) on the host cores
# ---------------------------------------------------------------------------
def reference_cpu_run(p, ub, seconds, threads=0):
    """One bounded run of the reference's own multicore B&B; returns
    (nodes/s, nodes, walltime, threads)."""
    import oracle
    if not oracle.reference_available():
        return None
    r = oracle.run_reference_bb(p, ub=ub, bound_mode=BOUND_MODE, branch_mode=BRANCH_MODE, threads=threads,
                                johnson=True, time_limit=seconds, timeout=seconds * 4 + 120)
    if "decomposed" not in r or not r.get("walltime"):
        return None
    return r["decomposed"] / r["walltime"], r["decomposed"], r["walltime"]


def host_cores():
    return os.cpu_count() or 1


# ---------------------------------------------------------------------------
# clocks during the timed region
# ---------------------------------------------------------------------------
class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def __enter__(self):
        fd, self.path = tempfile.mkstemp(prefix="clocks_", suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.QUERY,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self):
        rows = []
        try:
            for line in open(self.path):
                f = [x.strip() for x in line.split(",")]
                if len(f) >= 9 and f[1].isdigit():
                    rows.append(f)
        except OSError:
            pass
        finally:
            if self.path and os.path.exists(self.path):
                os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unavailable"]}
        sm = [int(r[1]) for r in rows]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i].lower() == "active"})
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": int(rows[0][2]), "reasons": reasons,
                "samples": len(rows)}


# ---------------------------------------------------------------------------
# factoradic slices of the permutation space, one per rank
# ---------------------------------------------------------------------------
def rank_slice(n, rank, world):
    """(pos, end) factoradic vectors of rank's share of the first level:
    the n root cells are split into contiguous blocks, one per rank.  A rank
    left without a cell (world > n) gets an empty interval (pos after end)."""
    if world == 1:
        return None
    per = [n // world + (1 if r < n % world else 0) for r in range(world)]
    lo = sum(per[:rank])
    hi = lo + per[rank] - 1
    rest = [n - 1 - i for i in range(1, n)]
    if per[rank] == 0:
        return [n - 1] + [0] * (n - 1), [0] + rest
    pos = [lo] + [0] * (n - 1)
    end = [hi] + rest
    return pos, end


def exchange_incumbent(dist, cost, device):
    """The ranks' only exchange: the best makespan known anywhere (4-byte
    MIN all-reduce; NCCL on GPUs, gloo in the CPU tests)."""
    import torch
    t = torch.tensor([int(cost)], dtype=torch.int32, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MIN)
    return int(t.item())


def run_ours(args):
    import numpy as np
    import torch
    import pbbperm_b200 as pb

    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    dist = None
    if ws > 1:
        import torch.distributed as dist
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=300))
    p = pb.synthetic_instance(SEED, N_JOBS, N_MACH)
    ub, _ = pb.neh(p)
    cfg = pb.Config(boundingMode=BOUND_MODE, adaptiveBranchingMode=BRANCH_MODE, nbIVMs=NB_IVMS, device=local,
                    warps_per_cta=args.warps_per_cta)
    eng = pb.Engine(p, cfg)
    sl = rank_slice(N_JOBS, rank, ws)
    if sl is None:
        eng.start(ub=ub)
    else:
        eng.start_interval(ub=ub, pos=sl[0], end=sl[1])

    def window():
        t0 = eng.result()
        done = eng.explore(args.window)
        t1 = eng.result()
        return t1["decomposed"] - t0["decomposed"], t1["device_seconds"] - t0["device_seconds"], done, t1

    from pbbperm_b200 import distributed as pdist
    root = list(range(N_JOBS))

    def exchange_ub(res, done=False):
        """Between windows: the incumbent (MIN all-reduce), then rebalancing
        -- an idle rank takes half of the busiest rank's intervals."""
        if dist is None:
            return
        best = exchange_incumbent(dist, res["cost"], "cuda")
        eng.set_ub(best)
        pdist.rebalance(dist, eng, N_JOBS, best, root, device="cuda", done=done)

    for _ in range(args.warmup):
        _, _, done, res = window()
        exchange_ub(res, done)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    nodes = 0
    dev_s = 0.0
    launches = 0
    steps_done = 0
    with ClockSampler(local) as clk:
        wall0 = time.perf_counter()
        for _ in range(args.steps):
            dn, ds, done, res = window()
            nodes += dn
            dev_s += ds
            launches += 1          # the explorer kernel (explorers persist across launches)
            steps_done += 1
            exchange_ub(res, done)
        torch.cuda.synchronize()
        wall = time.perf_counter() - wall0
    if dist:
        dist.barrier()
    clocks = clk.summary()
    res = eng.result()
    kern = eng.kernel_stats()
    eng.close()

    # whole-job aggregate: nodes summed, time = max over ranks
    tot_nodes, max_s = nodes, dev_s
    if dist:
        t = torch.tensor([float(nodes), dev_s], dtype=torch.float64, device="cuda")
        a = t.clone()
        dist.all_reduce(a[:1], op=dist.ReduceOp.SUM)
        b = t[1:].clone()
        dist.all_reduce(b, op=dist.ReduceOp.MAX)
        tot_nodes, max_s = a[0].item(), b[0].item()
    value = tot_nodes / max_s if max_s > 0 else 0.0

    # e2e through the C ABI from host buffers: every rank creates an engine on
    # its own slice (instance upload, tables, root + unfold), explores one
    # window and reads the result back; nodes are summed over ranks and the
    # step time is the slowest rank's
    e2e_vals = []
    for _ in range(args.e2e_steps):
        if dist:
            dist.barrier()
        t0 = time.perf_counter()
        with pb.Engine(p, cfg) as e2:
            if sl is None:
                e2.start(ub=ub)
            else:
                e2.start_interval(ub=ub, pos=sl[0], end=sl[1])
            e2.explore(args.window)
            r2 = e2.result()
        el = time.perf_counter() - t0
        nodes2, el2 = float(r2["decomposed"]), el
        if dist:
            t = torch.tensor([nodes2, el2], dtype=torch.float64, device="cuda")
            a = t[:1].clone()
            dist.all_reduce(a, op=dist.ReduceOp.SUM)
            b = t[1:].clone()
            dist.all_reduce(b, op=dist.ReduceOp.MAX)
            nodes2, el2 = a[0].item(), b[0].item()
        e2e_vals.append(nodes2 / el2)

    out = None
    if rank == 0:
        # processing times, Johnson entries and positions, pair machines, minimum
        # times, bound, root
        h2d = int(p.size * 4 + N_JOBS * 192 * 9 + 2 * 192 + 2 * N_MACH * 4 + 4 + 64 * 4)
        d2h = int(160 + 64)
        e2e = {"value": round(statistics.median(e2e_vals), 1) if e2e_vals else None, "unit": "nodes/s",
               "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
               "note": "per rank: engine creation + root/unfold + one window + result, summed over ranks, "
                       "time = slowest rank"}

        # roofline of the explorer kernel.  `achieved` = the INT32 operations of
        # the bounds as the explorer executes them (Engine.kernel_stats), per
        # second of its device time.  `equivalent` is the rate at which the
        # reference's formulation would have to run to keep up: 5m per weak child
        # ("m*(3 add+2 max)", bounds/src/bound_fsp_weak.cpp:132) and 4 P n + P per
        # Johnson child (add, add-lag, max, add per job and pair over the full
        # Johnson order, then the pair's close, bound_fsp_strong.cpp:84-100).  It
        # is no fraction of the peak: the explorer does not execute it.
        peak = pb.int32_peak(local)
        P = N_MACH * (N_MACH - 1) // 2
        algo_ops = kern["simple_bounds"] * 5.0 * N_MACH + kern["johnson_bounds"] * (4.0 * P * N_JOBS + P)
        secs = kern["device_seconds"]
        equivalent = algo_ops / secs / 1e9 if secs > 0 else 0.0
        achieved = kern["int32_ops"] / secs / 1e9 if secs > 0 else 0.0
        roofline = {"bound": "int32", "achieved": round(achieved, 1), "peak": round(peak, 1), "unit": "Gop/s",
                    "frac": round(achieved / peak, 4) if peak else None,
                    # DRAM bytes of one explorer launch: 1.98 GB in a 50 ms window of one
                    # ncu capture of this workload, scaled to this window by device time
                    "traffic": round(NCU_DRAM_BYTES_PER_S * args.window),
                    "traffic_unit": "bytes per launch",
                    "peak_source": "measured: pbb_diag_int32_peak (IADD+IMNMX register chains, all SMs)",
                    "work_model": kern["work_model"],
                    "equivalent": {"rate": round(equivalent, 1),
                                   "work_model": "simple LBs x 5m + Johnson LBs x (4 P n + P), P = m(m-1)/2"}}
        cpu = None
        if ws == 1 and args.cpu_sample > 0:
            r = reference_cpu_run(p, ub, args.cpu_sample)
            if r:
                cpu = {"value": round(r[0], 1), "unit": "nodes/s", "cores": host_cores(), "kind": "reference",
                       "sample": "oracle/_ref/bbJ (reference multicore, Johnson call restored) on the same "
                                 "instance/UB/modes, threads = all host cores, %.0f s window" % args.cpu_sample}
        extra = {}
        if ws == 1 and args.config2:
            extra["config2"] = run_config2(local)
        if ws == 1 and args.mode1:
            extra["mode1"] = run_mode1(local)
        if ws == 1 and args.summary_batch > 0:
            extra["batch"] = compact_batch(args.summary_batch, local)
        if ws == 1 and args.summary_serve > 0:
            extra["serve"] = compact_serve(args.summary_serve, args.summary_rate, local)
        out = {"metric": METRIC, "value": round(value, 1), "unit": "nodes/s", "n_gpus": ws, "steps": steps_done,
               "warmup": args.warmup, "ms_per_step": round(max_s / max(1, steps_done) * 1e3, 3),
               "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
               "data": "synthetic (seeded splitmix64 U[1,99])",
               "config": workload_config({"window_s": args.window, "parallelism": "dp%d" % ws if ws > 1 else "single"}),
               "e2e": e2e, "gpu_launches": launches, "clocks": clocks, "roofline": roofline,
               "cpu_baseline": cpu, "wall_s": round(wall, 3), "best_makespan": res["cost"],
               "counters": {"decomposed": res["decomposed"], "johnson_bounds": res["johnson_bounds"],
                            "simple_bounds": res["simple_bounds"], "leaves": res["leaves"],
                            "steals": res["steals"]}}
        out.update(extra)
    if dist:
        dist.barrier()
        dist.destroy_process_group()
    if out:
        print(json.dumps(out), flush=True)


def config2_golden():
    """Reference counters of the second configuration, if the fixture holds them."""
    path = os.path.join(ROOT, "tests", "golden", "search_golden.json")
    try:
        with open(path) as f:
            runs = json.load(f)["runs"]
    except (OSError, ValueError, KeyError):
        return None
    big = [r for r in runs if r.get("big")]
    return big[0] if big else None


def run_config2(device):
    """Second configuration: 20 jobs x 20 machines (seed 1), weak then Johnson,
    MinMin, UB = its optimum 2352, 16384 explorers, solved to completion (a
    narrow tree: the regime where work sharing, not the bound, limits speed).
    Counters are deterministic and checked against the reference's."""
    import pbbperm_b200 as pb
    p = pb.synthetic_instance(1, 20, 20)
    cfg = pb.Config(boundingMode=BOUND_MODE, adaptiveBranchingMode=BRANCH_MODE, nbIVMs=16384, device=device)
    runs = []
    for _ in range(3):
        with pb.Engine(p, cfg) as e:
            runs.append(e.solve(ub=2352))
    best = min(runs, key=lambda r: r["device_seconds"])
    g = config2_golden()
    keys = ("decomposed", "johnson_bounds", "simple_bounds", "leaves")
    exact = None if g is None else all(r[k] == g[k] for r in runs for k in keys)
    return {"workload": "pfsp-20x20-u1-99-seed1, UB = 2352 (optimum), 16384 explorers, to completion",
            "device_seconds": round(best["device_seconds"], 4),
            "nodes_per_s": round(best["decomposed"] / best["device_seconds"], 1) if best["device_seconds"] else None,
            "decomposed": best["decomposed"], "complete": all(r["complete"] for r in runs),
            "counters_equal_reference": exact, "runs": len(runs),
            "device_seconds_all": [round(r["device_seconds"], 4) for r in runs]}


def run_mode1(device, windows=3, window_s=2.0):
    """The bench workload with the Johnson bound on every child (boundingMode
    1: no weak pre-filter, the side chosen on the Johnson values), MinMin,
    UB = NEH, 65,536 explorers: decomposed nodes/s and Johnson bounds/s over
    fixed device-time windows after one warm-up window."""
    import pbbperm_b200 as pb
    p = pb.synthetic_instance(SEED, N_JOBS, N_MACH)
    ub = pb.neh(p)[0]
    cfg = pb.Config(boundingMode=1, adaptiveBranchingMode=BRANCH_MODE, nbIVMs=NB_IVMS, device=device)
    with pb.Engine(p, cfg) as e:
        e.start(ub=ub)
        e.explore(window_s)
        r0 = e.result()
        for _ in range(windows):
            e.explore(window_s)
        r1 = e.result()
    dt = r1["device_seconds"] - r0["device_seconds"]
    nodes = r1["decomposed"] - r0["decomposed"]
    jb = r1["johnson_bounds"] - r0["johnson_bounds"]
    return {"workload": "pfsp-50x20-u1-99-seed2, boundingMode 1 (Johnson on every child), MinMin, UB = NEH, "
                        "65536 explorers, %d x %.0f s windows" % (windows, window_s),
            "nodes_per_s": round(nodes / dt, 1) if dt > 0 else None,
            "johnson_bounds_per_s": round(jb / dt, 1) if dt > 0 else None,
            "device_seconds": round(dt, 3)}


# the pool shape the autotuner picks on the batched workload (bench.py
# --workload batch): 8-warp CTAs in the bulk, 20-warp CTAs for the tail
SUMMARY_POOL = dict(max_jobs=22, max_machines=20, warps_per_cta=8, tail_warps=0, window_s=0.02)


def compact_batch(count, device):
    """Batched form, compact: the first `count` instances of the batched
    workload through one pool against the same instances one at a time
    (single-instance engine, 16384 explorers), both from device NEH."""
    import pbbperm_b200 as pb
    from pbbperm_b200 import workloads
    r = workloads.run_batch(count, pool_config=pb.PoolConfig(device=device, **SUMMARY_POOL), device=device)
    return {"workload": "first %d instances of the batched workload (n 12-20, m 5/10/20, seeds 100+)" % count,
            "batch_inst_per_s": round(r["batch_inst_per_s"], 2), "one_at_a_time_inst_per_s":
            round(r["solo_inst_per_s"], 2), "speedup": round(r["speedup"], 2),
            "all_verified": r["all_verified"], "same_optima": r["same_optima_as_solo"], "pool": r["pool"]}


def compact_serve(count, rate, device):
    """Served form, compact: `count` requests of the Poisson stream at `rate`
    through the pool (continuous batching) and through a one-slot pool,
    latency = completion - arrival, NEH computed on the device per request."""
    import pbbperm_b200 as pb
    from pbbperm_b200 import workloads
    pc = pb.PoolConfig(device=device, **dict(SUMMARY_POOL, window_s=0.002))
    mix = workloads.serve_stream(rate, count, pool_config=pc, device=device)
    one = workloads.serve_stream(rate, count, pool_config=pc, device=device, max_resident=1)
    row = {"workload": "serve-poisson-n10-22-m5-20, %d requests at %g req/s" % (count, rate)}
    for name, r in (("mix", mix), ("one_at_a_time", one)):
        row[name] = {"throughput": round(r["throughput"], 2), "p50_ms": round(r["p50_ms"], 2),
                     "p99_ms": round(r["p99_ms"], 2), "all_verified": r["all_verified"]}
    row["speedup"] = round(mix["throughput"] / one["throughput"], 2)
    row["same_results_alone_and_in_mix"] = all(one["costs"][i] == mix["costs"][i] for i in mix["costs"])
    return row


def run_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0:
        return
    import oracle
    from pbbperm_b200.instances import synthetic_instance
    if not oracle.reference_available():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref not built (python oracle/build_ref.py)"}))
        return
    p = synthetic_instance(SEED, N_JOBS, N_MACH)
    ub, _ = oracle.Oracle(p).neh()
    step_s = min(args.window, 8.0)
    for _ in range(args.warmup):
        reference_cpu_run(p, ub, 2.0)
    vals = []
    t0 = time.perf_counter()
    for _ in range(args.steps):
        r = reference_cpu_run(p, ub, step_s)
        if r:
            vals.append(r[0])
    wall = time.perf_counter() - t0
    value = statistics.median(vals) if vals else 0.0
    out = {"impl": "reference", "metric": METRIC, "value": round(value, 1), "unit": "nodes/s", "n_gpus": ws,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(wall / max(1, args.steps) * 1e3, 3),
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int32",
           "data": "synthetic (seeded splitmix64 U[1,99])", "config": workload_config({"window_s": step_s}),
           "cpu_baseline": {"value": round(value, 1), "unit": "nodes/s", "cores": host_cores(), "kind": "reference",
                            "sample": "oracle/_ref/bbJ, all host threads, %.0f s window per step" % step_s},
           "e2e": {"value": round(value, 1), "unit": "nodes/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)


def run_batch_bench(args):
    """Batched configuration: autotune the pool on a calibration sample, solve
    all instances through one pool, compare with one-at-a-time solving."""
    import torch
    import pbbperm_b200 as pb
    from pbbperm_b200 import workloads, autotune
    from pbbperm_b200.instances import batch_instance
    torch.cuda.set_device(0)
    insts = [batch_instance(100 + i) for i in range(args.batch_count)]
    ubs = [pb.UB_NEH] * len(insts)
    t0 = time.perf_counter()
    pc, trials = autotune.tune_pool(insts, ubs, workloads.SEARCH, max_jobs=20, max_machines=20, repeats=1)
    t_tune = time.perf_counter() - t0
    if args.pool_window > 0:
        pc.window_s = args.pool_window
    r = workloads.run_batch(args.batch_count, pool_config=pc, solo_sample=args.batch_solo)
    out = {"metric": "batched solve throughput (instances/s)", "value": round(r["batch_inst_per_s"], 2),
           "unit": "instances/s", "n_gpus": 1, "higher_is_better": True,
           "config": {"workload": "batch-%d-uneven-n12-20-m5-10-20-seeds100+" % args.batch_count,
                      "bounding_mode": 2, "initial_ub": "NEH on the device (inside the timed solve)",
                      "pool": r["pool"]},
           "one_at_a_time": {"value": round(r["solo_inst_per_s"], 2), "unit": "instances/s",
                             "sample": r["solo_instances"], "engine_explorers": 16384},
           "speedup_vs_one_at_a_time": round(r["speedup"], 2), "batch_seconds": round(r["batch_seconds"], 3),
           "all_optima_verified": r["all_verified"], "same_optima_as_one_at_a_time": r["same_optima_as_solo"],
           "decomposed_nodes": r["nodes"], "autotune": {"seconds": round(t_tune, 2), "trials": trials}}
    print(json.dumps(out), flush=True)


def run_serve_bench(args):
    """Serving configuration: Poisson request streams through the pool
    (continuous batching) against the same streams served one request at a
    time through the same pool (max_resident = 1: no concurrency, no
    allocation per request), both measured end to end with p50/p99 latency;
    plus the service time of the single-instance engine (create + solve +
    destroy) on a sample of the requests."""
    import torch
    from pbbperm_b200 import workloads
    torch.cuda.set_device(0)
    rows = []
    for rate in [float(x) for x in args.rates.split(",")]:
        count = max(20, min(args.serve_requests, int(rate * args.serve_seconds)))
        mix = workloads.serve_stream(rate, count)
        one = workloads.serve_stream(rate, count, max_resident=1)
        same = all(one["costs"][i] == mix["costs"][i] for i in mix["costs"])
        row = {"rate": rate, "requests": count}
        for name, r in (("mix", mix), ("alone", one)):
            row[name] = {"throughput": round(r["throughput"], 2), "p50_ms": round(r["p50_ms"], 2),
                         "p99_ms": round(r["p99_ms"], 2), "all_verified": r["all_verified"]}
        row["speedup"] = round(mix["throughput"] / one["throughput"], 2)
        row["same_results_alone_and_in_mix"] = same
        rows.append(row)
        print(json.dumps(row), file=sys.stderr, flush=True)
    service, _ = workloads.alone_service(args.solo_sample)
    best = max(rows, key=lambda x: x["mix"]["throughput"])
    out = {"metric": "served solves/s with p50/p99 latency (continuous batching)",
           "value": best["mix"]["throughput"], "unit": "requests/s", "n_gpus": 1, "higher_is_better": True,
           "config": {"workload": "serve-poisson-n10-22-m5-20", "bounding_mode": 2,
                      "initial_ub": "NEH on the device (inside each request's latency)", "window_s": 0.002,
                      "requests_per_rate": "min(%d, rate x %g s)" % (args.serve_requests, args.serve_seconds)},
           "one_at_a_time": {"throughput": best["alone"]["throughput"], "kind": "same pool, one resident"},
           "speedup_vs_one_at_a_time": best["speedup"],
           "engine_per_request": {"requests": len(service), "mean_service_ms": round(1e3 * statistics.mean(service), 2),
                                  "capacity_req_per_s": round(len(service) / sum(service), 2)},
           "sweep": rows}
    print(json.dumps(out), flush=True)


if __name__ == "__main__":
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    elif a.workload == "batch":
        run_batch_bench(a)
    elif a.workload == "serve":
        run_serve_bench(a)
    else:
        run_ours(a)
