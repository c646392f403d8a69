#!/usr/bin/env python3
"""Benchmark of the superstep engine on the CC + SSSP workload at scale.

Workload (one step): on an undirected R-MAT graph of scale 24 (2^24 vertices,
edge factor 16, a/b/c/d = 0.57/0.19/0.19/0.05, seed 1, self-loops and
duplicates removed, symmetrised, u32 ids, u32 weights uniform in [1, 255]),
  - min-label connected components with the spread version (app cc), and
  - single-source shortest paths from vertex 0 with atomicMin delivery
    (app sssp_weighted, spread version),
each to quiescence, each run one captured CUDA-graph launch.  Metric:
Graph500-style GTEPS = stored edges x runs / time.  `value` times the runs
with the graph resident in HBM; `e2e` times the same through the C ABI with
host buffers (graph upload and result download inside the timed region).  Inputs are 3.8 GB, larger than the 126 MB L2, so no
L2 flush is needed between steps.

At N=1 the line also carries the other workloads (--no-extra skips them):
PageRank's precision split (FP32 compensated vs FP64, directed R-MAT scale
25, 30 rounds), the batched launch of 4,096 ER graphs against the per-graph
loop, and the request server on 16 resident graphs against the plain loop.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

With --gpus N > 1 (torchrun), every rank runs the same workload on its own GPU
(replicas: the path does not shard), and value is the sum over ranks.
"""
import argparse
import ctypes
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

METRIC = "PageRank/CC/SSSP GTEPS + HBM GB/s; served queries/s, p50/p99 vs plain GPU loop"
HBM_FALLBACK_GBS = 6650.0


def parse_args():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=5)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", default="ours", choices=["ours", "reference"])
    p.add_argument("--scale", type=int, default=24)
    p.add_argument("--no-e2e", action="store_true")
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--no-parity", action="store_true", help="skip the check of the results against the reference")
    p.add_argument("--write-traffic", nargs=2, metavar=("NCU_CSV", "BENCH_LINE"),
                   help="write profiles/traffic.json from an ncu launch list and the bench line of the same command")
    p.add_argument("--no-extra", action="store_true",
                   help="skip the PageRank precision-split, batched and serving workloads")
    p.add_argument("--rows", default="",
                   help="comma list of the other workloads to run (pagerank_precision_split, batched_many_graph, "
                        "serving); default all")
    return p.parse_args()


def dist_setup(n_gpus):
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def reduce_max(x, world, device):
    """Max of a float over the ranks of the default process group (the timing
    rule: a multi-GPU time is the slowest rank's)."""
    if world == 1:
        return float(x)
    import torch
    import torch.distributed as dist
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_gteps(world, edges_per_rank_run, runs, ms_max):
    """Whole-job Graph500 GTEPS of `world` replicas, each processing the same
    graph `runs` times, over the slowest rank's time."""
    return world * edges_per_rank_run * runs / (ms_max * 1e-3) / 1e9


def parse_clock_csv(path):
    """Median SM clock, max clock and throttle reasons seen in an nvidia-smi
    --query-gpu CSV (ClockSampler.FIELDS, noheader, nounits)."""
    sm, mx, reasons = [], None, set()
    names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
    for line in open(path):
        parts = [x.strip() for x in line.split(",")]
        if len(parts) < 9:
            continue
        try:
            sm.append(float(parts[1]))
            mx = float(parts[2])
        except ValueError:
            continue
        for n, v in zip(names, parts[5:9]):
            if v.lower() == "active":
                reasons.add(n)
    return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
            "samples": len(sm)}


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return HBM_FALLBACK_GBS, "fallback"


NVML_REASONS = (("hw_slowdown", 0x8), ("sw_thermal_slowdown", 0x20), ("hw_thermal_slowdown", 0x40),
                ("sw_power_cap", 0x4))


def nvml_reasons(mask):
    return [n for n, bit in NVML_REASONS if mask & bit]


class ClockSampler:
    """SM clock and clock-event reasons during the timed region: NVML read
    queries every 10 ms on a thread (the timed regions are a fraction of a
    second), else nvidia-smi every 200 ms.  Reads only; no setting changes."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    PERIOD_S = 0.01

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.path = None
        self.thread = None
        self.samples = []
        self.mask = 0
        self.max_mhz = None

    def _nvml_handle(self):
        import pynvml
        import torch
        pynvml.nvmlInit()
        p = torch.cuda.get_device_properties(self.gpu)
        bus = f"{p.pci_domain_id:08X}:{p.pci_bus_id:02X}:{p.pci_device_id:02X}.0"
        return pynvml, pynvml.nvmlDeviceGetHandleByPciBusId(bus)

    def start(self):
        import threading
        try:
            nv, h = self._nvml_handle()
            self.max_mhz = float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM))
            self.stop_flag = threading.Event()

            def run():
                while not self.stop_flag.is_set():
                    try:
                        self.samples.append(float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)))
                        self.mask |= int(nv.nvmlDeviceGetCurrentClocksEventReasons(h))
                    except Exception:
                        pass
                    self.stop_flag.wait(self.PERIOD_S)

            self.thread = threading.Thread(target=run, daemon=True)
            self.thread.start()
            return
        except Exception:
            self.thread = None
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.thread is not None:
            self.stop_flag.set()
            self.thread.join(timeout=5)
            return {"sm_mhz": statistics.median(self.samples) if self.samples else None,
                    "sm_max_mhz": self.max_mhz, "reasons": nvml_reasons(self.mask),
                    "samples": len(self.samples), "source": "NVML, 10 ms"}
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        out = parse_clock_csv(self.path)
        out["source"] = "nvidia-smi, 200 ms"
        os.unlink(self.path)
        return out


def cpu_host_info():
    model = "unknown"
    try:
        for line in open("/proc/cpuinfo"):
            if line.startswith("model name"):
                model = line.split(":", 1)[1].strip()
                break
    except Exception:
        pass
    return os.cpu_count() or 1, model


REF_ENV_NOTE = "OMP_PROC_BIND=TRUE, OMP_PLACES=cores, schedule static, chunk 0 (submission.slurm:36-42)"


def reference_run(app, graph_path, threads, dump=True):
    """One run of the reference's own OpenMP binary <app>_spread_32 (oracle/_ref)
    on graph files, with all host threads and the environment of
    submission.slurm:36-42.  Returns (the reference's own "Total time of
    supersteps" in seconds, its dump text or None, its stdout).  The dump goes
    to /dev/null when not needed (the dump is outside the timed supersteps)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    env = {"OMP_NUM_THREADS": str(threads), "OMP_PROC_BIND": "TRUE", "OMP_PLACES": "cores"}
    if dump:
        text, out = O.run_ref(app, "spread", graph_path, threads=threads, schedule="static", chunk=0, env=env,
                              timeout=1800)
    else:
        _, out = O.run_ref(app, "spread", graph_path, threads=threads, schedule="static", chunk=0, env=env,
                           timeout=1800, dump=False)
        text = None
    return O.parse_total_time(out), text, out


def reference_arm(args, rank, world):
    """The reference's own CPU implementation of the path, on this arm's
    workload: the scale-24 undirected R-MAT graph, generated by the oracle's
    CPU generator (the same CSR as the device generator) and written once in
    the reference loader's format.  Step k runs cc_spread_32 (k even) or
    sssp_spread_32 (k odd), so that the K + W runs end within minutes; each
    run's time is the reference's own "Total time of supersteps".  The
    reference's SSSP counts hops: weighted SSSP has no reference
    implementation.  Nothing of this repository's GPU runtime is loaded."""
    if rank != 0:
        return 0
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    if not O.have_ref():
        print(json.dumps({"impl": "reference", "unavailable": "reference binaries (oracle/_ref) were not built"}))
        return 0
    scale = args.scale
    t_gen = time.time()
    g = O.gen_rmat(scale, 16, seed=1, undirected=True)
    t_gen = time.time() - t_gen
    V, E = g.V, g.E
    cores, model = cpu_host_info()
    per = {"cc": [], "sssp": []}
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, f"rmat{scale}")
        O.write_graph(g, path)
        del g
        apps = ("cc", "sssp")
        for k in range(args.warmup):
            reference_run(apps[k % 2], path, cores, dump=False)
        secs = []
        for k in range(args.steps):
            t, _, _ = reference_run(apps[k % 2], path, cores, dump=False)
            per[apps[k % 2]].append(t)
            secs.append(t)
    value = E * len(secs) / sum(secs) / 1e9
    per_prog = {a: {"runs": len(v), "best_s": round(min(v), 4), "mean_s": round(sum(v) / len(v), 4),
                    "gteps_best": round(E / min(v) / 1e9, 4)} for a, v in per.items() if v}
    workload = (f"cc (spread) + sssp (spread, hop count: the reference has no weighted SSSP), undirected R-MAT "
                f"scale {scale}, edge factor 16, a/b/c=0.57/0.19/0.19, seed 1")
    sample = (f"reference cc_spread_32 and sssp_spread_32 (oracle/_ref, compiled from the reference sources) on the "
              f"scale-{scale} graph (V={V}, E={E}, generated by the oracle's CPU generator in {t_gen:.0f} s, "
              f"untimed), steps alternate the two programs, {cores} OpenMP threads, {REF_ENV_NOTE}, "
              f"'Total time of supersteps', CPU {model}")
    line = {
        "metric": METRIC, "value": round(value, 4), "unit": "GTEPS", "impl": "reference", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(1e3 * sum(secs) / len(secs), 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
        "config": {"workload": workload, "vertices": V, "edges_stored": E,
                   "teps": "Graph500: stored edges per run / superstep time",
                   "step": "one reference run: cc_spread_32 on even steps, sssp_spread_32 on odd steps"},
        "per_program": per_prog,
        "cpu_baseline": {"value": round(value, 4), "unit": "GTEPS", "cores": cores, "kind": "reference",
                         "sample": sample},
        "e2e": {"value": round(value, 4), "unit": "GTEPS", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


def pagerank_row(peak, check_oracle=True):
    """PageRank precision split on directed R-MAT scale 25, 30 rounds: FP32
    compensated pull (ipg_pr_run_f32) against the FP64 engine (pagerank,
    single broadcast), per-vertex error of FP32 against FP64 on the GPU."""
    import numpy as np
    import torch
    import ipregel_b200 as ip
    scale, rounds = 25, 30
    g = ip.Graph.generate_rmat(scale, 16, seed=1, undirected=False)
    g.set_directed(False)  # the stored rows are the gather lists, as the reference loads them
    V, E = g.V, g.E
    pr = ip.PageRankF32(g)
    x = ip.DeviceArray(V, np.float32)
    d = ip.DeviceArray((rounds + 1) * 3, np.float64)
    for _ in range(2):
        pr.run_device(x, d, rounds, 0.85, True)
    torch.cuda.synchronize()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    reps = 3
    t0.record()
    for _ in range(reps):
        pr.run_device(x, d, rounds, 0.85, True)
    t1.record()
    torch.cuda.synchronize()
    ms32 = t0.elapsed_time(t1) / reps
    diag = d.to_host().reshape(rounds + 1, 3)
    eng = ip.Engine("pagerank", "single_broadcast")
    eng.set_quiet(True)
    eng.set_param("rounds", rounds)
    eng.set_graph_loop(True)
    eng.attach(g)
    eng.run_only()
    ms64 = []
    for _ in range(2):
        eng.run_only()
        ms64.append(eng.stats()[0] * 1e3)
    eng_counts = eng.counts()
    ptr = ctypes.c_void_p()
    eng._check(eng.lib.ipg_app_values_device(ctypes.byref(ptr)), "ipg_app_values_device")
    err = ip.error_f32_f64(x, ip.DeviceArray.wrap(ptr.value, V, np.float64))
    v64 = eng.values()
    v32 = x.to_host()
    eng.set_graph_loop(False)
    eng.set_param("rounds", 10)
    eng.release()
    # both against the FP64 CPU oracle (pagerank single_broadcast, the same
    # 30 rounds on the same CSR), outside the timed runs
    vs_oracle = None
    if check_oracle:
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import oracle as O
        t_chk = time.time()
        idx, adj, _ = g.to_host()
        want, counts, _ = O.run(O.CSR(V, E, idx, adj), "pagerank", "single_broadcast", rounds=rounds)
        del idx, adj
        a64 = np.abs(v64 - want)
        a32 = np.abs(v32.astype(np.float64) - want)
        nz = want != 0
        vs_oracle = {"fp64_engine_max_abs": float(a64.max()), "fp64_within_1e-12": bool(a64.max() <= 1e-12),
                     "fp64_counts_equal": [int(c) for c in counts] == eng_counts,
                     "fp32_max_abs": float(a32.max()),
                     "fp32_max_rel": float((a32[nz] / want[nz]).max()) if nz.any() else 0.0,
                     "fp32_mean_abs": float(a32.mean()),
                     "oracle": "FP64 CPU restatement of pagerank.c's single_broadcast run (oracle/), "
                               f"{time.time() - t_chk:.0f} s"}
    byts = 8 * E + 24 * V
    achieved = byts / (ms32 / rounds * 1e-3) / 1e9
    launches = launches_per_run_f32(rounds)
    # the gathers' access pattern alone: one scattered 4-byte quotient per edge
    ceil = ip.measure_gather(4 * V, 4, 1 << 28, 5)
    edge_rate = E * rounds / (ms32 * 1e-3)
    out = {"workload": f"PageRank, directed R-MAT scale {scale}, edge factor 16, seed 1, {rounds} rounds, d=0.85",
           "vertices": V, "edges": E,
           "fp32_compensated": {"ms": round(ms32, 3), "gteps": round(E * rounds / (ms32 * 1e-3) / 1e9, 2),
                                "algorithmic_gbs": round(achieved, 1), "frac_hbm": round(achieved / peak, 4),
                                "bytes_per_superstep": "8E + 24V (ids, quotient gathers; row, value, quotient)",
                                "gpu_launches": launches,
                                "gather_ceiling": {
                                    "pattern": f"u32 index stream + one scattered 4-byte read per index, table "
                                               f"{4 * V >> 20} MiB (the quotients), ipg_measure_gather",
                                    "rows_per_s": round(ceil["rows_per_s"] / 1e9, 2),
                                    "edges_per_s": round(edge_rate / 1e9, 2), "unit": "G/s",
                                    "frac": round(edge_rate / ceil["rows_per_s"], 4) if ceil["rows_per_s"] else None}},
           "fp64_engine": {"ms": round(min(ms64), 3), "gteps": round(E * rounds / (min(ms64) * 1e-3) / 1e9, 2)},
           "fp32_vs_fp64": {k: (float(f"{v:.4g}") if isinstance(v, float) else v) for k, v in err.items()},
           "vs_fp64_cpu_oracle": vs_oracle,
           "fp64_diagnostics_last": {"mass": float(diag[-1, 0]), "dangling": float(diag[-1, 1]),
                                     "residual_l1": float(diag[-1, 2])}}
    x.free()
    d.free()
    pr.free()
    g.free()
    return out


def launches_per_run_f32(rounds):
    return 2 + rounds  # superstep 0, the rounds, the values in the caller's numbering


def batch_row():
    """4,096 directed ER graphs (n log-uniform in [1024, 65536], out-degree 8,
    weights U[1,64]): CC + SSSP(0) of every graph in one fused CUDA-graph
    launch after autotuning, against the plain loop (attach and run per graph)."""
    import numpy as np
    from ipregel_b200 import batch as B
    sizes = B.log_uniform_sizes(4096, 1024, 65536, seed=1)
    parts = B.generate_er_parts(sizes, degree=8, seed=1, wmax=64)
    bt = B.Batch(parts, directed=True)
    r = B.BatchRunner(bt)
    best = r.autotune()
    for _ in range(2):
        r.run()
    ts = [r.run() for _ in range(5)]
    res = r.results()
    fused = min(ts)
    launches = r.cc.launches() + r.sp.launches()
    pcc, psp, wall, dev = B.run_plain(parts)
    same = all(np.array_equal(pcc[i], res.cc[i]) and np.array_equal(psp[i], res.sssp[i]) for i in range(len(parts)))
    E = bt.union.E
    out = {"workload": "4096 directed ER graphs, n log-uniform [1024, 65536], m = 8n, weights U[1,64], seed 1; "
                       "CC + SSSP(0) per graph",
           "vertices": int(bt.union.V), "edges": int(E),
           "speedup_vs_plain_device": round(dev / fused, 1),
           "speedup_note": "device time of the fused launch against the device time of the plain per-graph loops; "
                           "the wall-clock ratio also counts the plain loop's host attach/run calls",
           "fused_launch_ms": round(fused * 1e3, 2), "fused_gteps_2runs": round(2 * E / fused / 1e9, 3),
           "plain_loop_device_s": round(dev, 3), "plain_loop_wall_s": round(wall, 3),
           "speedup_vs_plain_wall": round(wall / fused, 1),
           "results_equal_plain": bool(same),
           "tuning": {k: v[0] for k, v in best.items()}, "supersteps": list(res.supersteps)}
    r.release()
    bt.free()
    return out


def serving_row():
    """16 resident undirected R-MAT graphs, scales 18..25 (two each), weights
    U[1,255]; 2,000 queries with Poisson arrivals at 2,000/s, 60% SSSP, 30%
    PPR (FP32, 20 rounds), 10% CC; served throughput and latency, against the
    plain loop run serially on a sample of the same trace."""
    import numpy as np
    import torch
    import ipregel_b200 as ip
    from ipregel_b200 import serve as S
    scales = [s for s in range(18, 26) for _ in range(2)]
    graphs = [ip.Graph.generate_rmat(s, 16, seed=100 + i, undirected=True, wmax=255) for i, s in enumerate(scales)]
    sizes = [g.V for g in graphs]
    srv = S.Server(hbm_budget=0, ppr_rounds=20)
    for g in graphs:
        gid = srv.add_graph(g)
        for kind in (S.SSSP, S.PPR):  # per-query vertex state resident before the trace
            srv.reserve(gid, kind)
    srv.run_trace(S.poisson_trace(64, 2000.0, sizes, seed=99))
    tr = S.poisson_trace(2000, 2000.0, sizes, seed=1)
    free_b, total_b = torch.cuda.mem_get_info()
    # the trace three times: continuous batching is timing dependent (which
    # queries share a superstep), so served throughput varies from run to run;
    # the run with the median throughput is reported, all three beside it
    runs = []
    for _ in range(3):
        clocks = ClockSampler(torch.cuda.current_device())
        clocks.start()
        _, lat, mk = srv.run_trace(tr)
        clk = clocks.stop()
        runs.append((S.summarize(lat, mk, tr.kind), clk))
    runs.sort(key=lambda r: r[0]["qps"])
    summ, clk = runs[1]
    # below capacity: arrivals at about an eighth of the served rate, so that the
    # percentiles are service latencies rather than queueing
    low_rate = 40.0
    tr_low = S.poisson_trace(200, low_rate, sizes, seed=2)
    _, lat_low, mk_low = srv.run_trace(tr_low)
    low = S.summarize(lat_low, mk_low, tr_low.kind)
    st = srv.stats()
    # device time, supersteps and lanes per lane-group kind and graph scale
    groups = {}
    for gid, name, busy, steps, lanes, _ in srv.group_stats():
        a = groups.setdefault(f"scale{scales[gid]}:{name}", {"busy_s": 0.0, "supersteps": 0, "lanes": 0})
        a["busy_s"] = round(a["busy_s"] + busy, 3)
        a["supersteps"] += steps
        a["lanes"] += lanes
    for k, a in groups.items():
        if k.endswith(":ppr") and a["supersteps"]:
            a["mean_busy_lanes"] = round(a["lanes"] * 20 / a["supersteps"], 1)  # each lane runs 20 gathers
    srv.free()
    m = 150
    tot, per = 0.0, {0: [], 1: [], 2: []}
    engines = {S.SSSP: ("sssp_weighted", "spread"), S.PPR: ("ppr", "single_broadcast"), S.CC: ("cc", "spread")}
    for kind, (app, ver) in engines.items():
        eng = ip.Engine(app, ver)
        eng.set_quiet(True)
        if app == "ppr":
            eng.set_param("rounds", 20)
        for gid in range(len(graphs)):
            sel = [i for i in range(m) if tr.kind[i] == kind and tr.gid[i] == gid]
            if not sel:
                continue
            eng.attach(graphs[gid])
            for i in sel:
                if kind != S.CC:
                    eng.set_param("source", int(tr.source[i]))
                eng.run_only()
                sec = eng.stats()[0]
                tot += sec
                per[kind].append(sec)
        eng.release()
    plain_qps = m / tot
    for g in graphs:
        g.free()
    return {"workload": "16 undirected R-MAT graphs, scales 18-25 (two each), edge factor 16, weights U[1,255]; "
                        "2000 queries, Poisson 2000/s, 60% SSSP / 30% PPR FP32 20 rounds / 10% CC, seed 1",
            "served_qps": round(summ["qps"], 1), "served_qps_runs": [round(r[0]["qps"], 1) for r in runs],
            "p50_ms": round(summ["p50_ms"], 1), "p99_ms": round(summ["p99_ms"], 1),
            "per_kind_ms": {k: round(v, 1) for k, v in summ.items() if k.endswith("_ms") and "_" in k[:-3]},
            "plain_serial_qps": round(plain_qps, 1),
            "plain_sample": f"first {m} queries of the trace, run one at a time through the plain engine "
                            f"(sssp_weighted/spread, ppr/single_broadcast FP64, cc/spread), graph attached "
                            f"once per graph, device loop time only",
            "speedup_vs_plain": round(summ["qps"] / plain_qps, 2),
            "counters_cover": "the 64-query warm-up trace, the three runs and the unsaturated trace",
            "groups": groups,
            "groups_note": "per graph scale (two graphs each) and group kind: summed superstep device time "
                           "(concurrent groups overlap), supersteps, lanes admitted; PPR: mean busy lanes of 32",
            "lanes_admitted": st["lanes_admitted"], "supersteps": st["supersteps"],
            "kernel_launches": st["kernel_launches"], "pull_supersteps": st["pull_supersteps"],
            "peak_hbm_bytes": st["peak_bytes"], "hbm_free_before_trace": free_b, "clocks_during_trace": clk,
            "note": "arrivals exceed capacity: latency includes queueing",
            "unsaturated": {"workload": f"200 queries of the same mix, Poisson {low_rate:.0f}/s (an eighth of the "
                                        f"served rate), seed 2", "served_qps": round(low["qps"], 1),
                            "p50_ms": round(low["p50_ms"], 2), "p99_ms": round(low["p99_ms"], 2),
                            "per_kind_ms": {k: round(v, 2) for k, v in low.items()
                                            if k.endswith("_ms") and "_" in k[:-3]}}}


def same_work_row(args, cc, g, E, world, barrier, max_over_ranks):
    """CC (spread) + hop-count SSSP from 0 (spread: benchmarks/sssp.c's
    program) on the headline graph, resident, through the captured loop: the
    work the reference arm times, for a like-for-like ratio.  Returns (row,
    hop distances of the last run, per-superstep counts)."""
    import torch
    import ipregel_b200 as ip
    hop = ip.Engine("sssp", "spread")
    hop.set_quiet(True)
    hop.set_graph_loop(True)
    hop.attach(g)
    for _ in range(args.warmup):
        cc.run_only()
        hop.run_only()
    barrier()
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0.record()
    ms_cc = ms_hop = 0.0
    for _ in range(args.steps):
        cc.run_only()
        ms_cc += cc.stats()[0] * 1e3
        hop.run_only()
        ms_hop += hop.stats()[0] * 1e3
    t1.record()
    barrier()
    ms = max_over_ranks(t0.elapsed_time(t1))
    res, counts, steps = hop.values(), hop.counts(), hop.stats()[2]
    hop.release()
    row = {"workload": "cc (spread) + sssp (spread, hop count from 0: benchmarks/sssp.c) on the headline graph, "
                       "resident, captured loop",
           "value": round(replica_gteps(world, E, 2 * args.steps, ms), 4), "unit": "GTEPS",
           "ms_per_step": round(ms / args.steps, 3),
           "gteps_per_program": {"cc": round(E * args.steps / (ms_cc * 1e-3) / 1e9, 4),
                                 "sssp_hop": round(E * args.steps / (ms_hop * 1e-3) / 1e9, 4)},
           "supersteps_sssp_hop": steps}
    return row, res, counts


def cpu_baseline_leg(g, E):
    """The reference's own binaries (oracle/_ref cc_spread_32, sssp_spread_32)
    once each on the headline graph itself (written in the reference loader's
    format), all host threads: about 10-30 s of CPU work.  Returns (the
    cpu_baseline object, {app: (dump text, stdout)}) -- the dumps also serve
    the parity check."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    cores, model = cpu_host_info()
    if not O.have_ref():
        return {"value": None, "unit": "GTEPS", "cores": cores, "kind": "reference",
                "sample": "reference binaries not built"}, {}
    dumps, secs = {}, {}
    with tempfile.TemporaryDirectory() as td:
        path = os.path.join(td, "graph")
        g.write(path)
        for app in ("cc", "sssp"):
            t, text, out = reference_run(app, path, cores, dump=True)
            secs[app] = t
            dumps[app] = (text, out)
    total = sum(secs.values())
    cpu = {"value": round(2.0 * E / total / 1e9, 4), "unit": "GTEPS", "cores": cores, "kind": "reference",
           "sample": f"reference cc_spread_32 + sssp_spread_32 (hop-count SSSP; weighted SSSP has no reference "
                     f"implementation), one run each on the headline scale-24 graph (E={E}), {cores} OpenMP "
                     f"threads, {REF_ENV_NOTE}, 'Total time of supersteps', CPU {model}",
           "seconds": {k: round(v, 4) for k, v in secs.items()}}
    return cpu, dumps


def parity_check(V, E, idx, adj, wgt, res_cc, counts_cc, res_sp, res_hop, counts_hop, ref_dumps):
    """Checks the timed runs' results: CC labels and hop-count SSSP distances
    against the reference binaries' own dumps of the same graph (else the
    oracle's restatement), per-superstep active counts against the
    reference's log lines, weighted SSSP distances against the oracle's exact
    Dijkstra.  Bit-exact comparisons."""
    import numpy as np
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    t = time.time()
    g = O.CSR(V, E, idx, adj, wgt)
    out = {}
    for app, res, counts in (("cc", res_cc, counts_cc), ("sssp", res_hop, counts_hop)):
        if res is None:
            continue
        if app in ref_dumps:
            text, stdout = ref_dumps[app]
            want = O.parse_dump_fast(text, V)
            want_counts = O.parse_counts(stdout)
            against = f"reference {app}_spread_32 dump"
        else:
            want, want_counts, _ = O.run(g, app, "spread")
            want_counts = [int(c) for c in want_counts]
            against = f"oracle {app} spread"
        out[app] = {"values_equal": bool(np.array_equal(np.asarray(res, dtype=np.uint32), want)),
                    "counts_equal": [int(c) for c in counts] == list(want_counts), "against": against}
    d = O.dijkstra(g, 0)
    out["sssp_weighted"] = {"values_equal": bool(np.array_equal(np.asarray(res_sp, dtype=np.uint32), d)),
                            "against": "oracle Dijkstra (exact, integer)"}
    ok = all(v["values_equal"] and v.get("counts_equal", True) for v in out.values())
    return {"ok": ok, **out, "check_s": round(time.time() - t, 1)}


TRAFFIC_PATH = os.path.join(ROOT, "profiles", "traffic.json")
# The kernel sources a DRAM capture describes: the engine headers and the
# runtime's kernels.  A capture of other sources says nothing about these.
KERNEL_SOURCES = ("include/ipregel_b200/engine.cuh", "include/ipregel_b200/host.cuh",
                  "include/ipregel_b200/api.cuh", "ipregel_b200/csrc/runtime.cu")


def kernel_sources_sha16():
    import hashlib
    h = hashlib.sha256()
    for rel in KERNEL_SOURCES:
        with open(os.path.join(ROOT, rel), "rb") as f:
            h.update(f.read())
    return h.hexdigest()[:16]


def stored_traffic(name, bytes_per_launch):
    """roofline.traffic from profiles/traffic.json: the DRAM bytes per
    algorithmic byte that one ncu capture measured for this kernel, times
    this launch's algorithmic bytes -- only when that capture ran the same
    kernel sources as this build (else null, with the reason)."""
    try:
        d = json.load(open(TRAFFIC_PATH))
    except Exception:
        return {"traffic": None, "traffic_source": "no DRAM capture stored (profiles/traffic.json)"}
    if d.get("_kernel_sources_sha16") != kernel_sources_sha16():
        return {"traffic": None,
                "traffic_source": "the stored DRAM capture (profiles/traffic.json) ran other kernel sources "
                                  "than this build"}
    tr = d.get(name)
    if not tr:
        return {"traffic": None, "traffic_source": f"no DRAM capture of {name} stored"}
    return {"traffic": round(tr["dram_bytes_per_algorithmic_byte"] * bytes_per_launch),
            "traffic_source": "scaled, not measured by this run: DRAM/algorithmic bytes of this kernel in an ncu "
                              "capture of the same kernel sources (" + tr["source"] + "), times this launch's "
                              "algorithmic bytes"}


# kernels of the build, and of the launch lists of builds before it
NCU_KERNEL_NAMES = (("ipx_k_push<0>", "push_thread"), ("ipx_k_push<1>", "push_warp"), ("ipx_k_push<2>", "push_block"),
                    ("ipx_k_compute_spread", "compute"), ("ipx_k_front", "compute"), ("ipx_k_push(", "push"),
                    ("ipx_k_count(", "count_active"))
# a superstep's first launch
NCU_SUPERSTEP_OPENERS = ("ipx_k_begin_superstep", "ipx_k_front")


def write_traffic(csv_path, line_path, out_path=TRAFFIC_PATH):
    """profiles/traffic.json from an ncu launch list (--metrics
    gpu__time_duration.sum,dram__bytes_read.sum,dram__bytes_write.sum --csv)
    of `bench.py --steps 1 --warmup 1 --no-e2e --no-cpu-baseline --no-extra
    --no-parity` and the JSON line of the same command run without ncu (its
    `kernels` give the algorithmic bytes).  The profiled step runs CC, then
    SSSP, each superstep opening with one of NCU_SUPERSTEP_OPENERS; in lists of
    builds before the compute kernel listed the broadcasters itself, k_compact
    launches alternate broadcasters / next frontier within a superstep."""
    import csv
    line = json.loads(open(line_path).read().strip().splitlines()[-1])
    steps_cc = line["kernels"]["cc:compute"]["launches"]
    rows = [r for r in csv.DictReader(l for l in open(csv_path) if not l.startswith("=="))]
    launches = {}
    for r in rows:
        launches.setdefault(r["ID"], {"name": r["Kernel Name"]})[r["Metric Name"]] = float(r["Metric Value"].replace(",", ""))
    order = [launches[k] for k in sorted(launches, key=int)]
    # the profiled step: the last 2 runs' host-loop launches, from the first
    # superstep of its CC run
    begins = [i for i, x in enumerate(order) if x["name"].startswith(NCU_SUPERSTEP_OPENERS)]
    steps_sp = line["kernels"]["sssp:compute"]["launches"]
    begins = begins[-(steps_cc + steps_sp):]
    dram, seen = {}, {}
    for j, b in enumerate(begins):
        prog = "cc" if j < steps_cc else "sssp"
        end = begins[j + 1] if j + 1 < len(begins) else len(order)
        compacts = 0
        for x in order[b:end]:
            nm = x["name"]
            if nm.startswith("void "):  # templated kernels carry their return type
                nm = nm[5:]
            key = None
            for pref, short in NCU_KERNEL_NAMES:
                if nm.startswith(pref):
                    key = short
            if nm.startswith("k_compact"):
                key = "compact_broadcasters" if compacts == 0 else "compact_targets"
                compacts += 1
            if key is None:
                continue
            k = f"{prog}:{key}"
            dram[k] = dram.get(k, 0.0) + x.get("dram__bytes_read.sum", 0.0) + x.get("dram__bytes_write.sum", 0.0)
            seen[k] = seen.get(k, 0) + 1
    out = {"_kernel_sources_sha16": kernel_sources_sha16()}
    for k, b in sorted(dram.items(), key=lambda kv: -kv[1]):
        alg = line["kernels"].get(k, {}).get("bytes")
        if not alg:
            continue
        out[k] = {"dram_bytes_per_algorithmic_byte": round(b / alg, 4), "launches": seen[k], "dram_bytes": int(b),
                  "algorithmic_bytes": int(alg),
                  "source": f"ncu 1-pass dram__bytes_read.sum + dram__bytes_write.sum over one profiled CC + SSSP "
                            f"step, R-MAT scale {line['config'].get('scale', 24)}"}
    with open(out_path, "w") as f:
        json.dump(out, f, indent=1)
    return out


def main():
    args = parse_args()
    if args.write_traffic:
        print(json.dumps(write_traffic(*args.write_traffic), indent=1))
        return 0
    rank, world, local = dist_setup(args.gpus)
    if args.impl == "reference":
        return reference_arm(args, rank, world)

    import numpy as np
    import torch
    import torch.distributed as dist

    torch.cuda.set_device(local)
    if world > 1:
        from datetime import timedelta
        dist.init_process_group("nccl", timeout=timedelta(seconds=600))
    import ipregel_b200 as ip

    scale = args.scale
    g = ip.Graph.generate_rmat(scale, 16, seed=1, undirected=True, wmax=255)
    V, E = g.V, g.E
    cc = ip.Engine("cc", "spread")
    sp = ip.Engine("sssp_weighted", "spread")
    for eng in (cc, sp):
        eng.set_quiet(True)
        eng.set_graph_loop(True)  # each run: one captured CUDA-graph launch
    sp.set_param("source", 0)
    cc.attach(g)
    sp.attach(g)
    renamed = cc.order()  # the kernels run on the graph's degree-ordered copy

    def step():
        cc.run_only()
        sp.run_only()

    for _ in range(args.warmup):
        step()

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(x):
        return reduce_max(x, world, "cuda")

    # ---- device-resident timed region ----
    for eng in (cc, sp):
        eng.profile_reset()
    clocks = ClockSampler(local)
    clocks.start()
    barrier()
    t0 = torch.cuda.Event(enable_timing=True)
    t1 = torch.cuda.Event(enable_timing=True)
    t0.record()
    edges_traversed = 0
    supersteps = []
    for _ in range(args.steps):
        step()
        edges_traversed += cc.stats()[1] + sp.stats()[1]
        supersteps.append((cc.stats()[2], sp.stats()[2]))
    t1.record()
    barrier()
    clk = clocks.stop()
    ms = max_over_ranks(t0.elapsed_time(t1))
    launches = cc.launches() + sp.launches()
    # the timed runs' own results, checked after the timing against the
    # reference's binaries and the oracle (parity)
    res_cc, res_sp = cc.values(), sp.values()
    counts_cc = cc.counts()

    runs = 2 * args.steps
    value = replica_gteps(world, E, runs, ms)
    traversed_gteps = world * edges_traversed / (ms * 1e-3) / 1e9

    # ---- one profiled step (host-driven loop, events around every launch) ----
    for eng in (cc, sp):
        eng.set_graph_loop(False)
        eng.set_profile(True)
        eng.profile_reset()
    step()
    prof = {}
    for tag, eng in (("cc", cc), ("sssp", sp)):
        for k, v in eng.profile().items():
            prof[f"{tag}:{k}"] = v
    for eng in (cc, sp):
        eng.set_profile(False)
        eng.set_graph_loop(True)  # every later run (same-work row, e2e) is one captured launch again

    # dominant kernel and its roofline
    peak, peak_kind = measured_peaks()
    top = max(prof.items(), key=lambda kv: kv[1]["ms"])
    top_name, top_rec = top
    avg_ms = top_rec["ms"] / max(top_rec["timed"], 1)
    bytes_per_launch = top_rec["bytes"] / max(top_rec["timed"], 1)
    achieved = bytes_per_launch / (avg_ms * 1e-3) / 1e9 if avg_ms > 0 else 0.0
    total_kernel_ms = sum(v["ms"] for v in prof.values())
    roofline = {"bound": "hbm", "kernel": top_name, "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                "frac": round(achieved / peak, 4), "traffic": None,
                "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)" if peak_kind == "measured" else peak_kind,
                "bytes_per_launch": round(bytes_per_launch), "avg_launch_ms": round(avg_ms, 4),
                "share_of_kernel_time": round(top_rec["ms"] / total_kernel_ms, 3) if total_kernel_ms else None,
                "timing": "CUDA events around each launch of one separate profiled step"}
    edges_per_launch = top_rec.get("edges", 0.0) / max(top_rec["timed"], 1)
    if edges_per_launch > 0 and avg_ms > 0:
        # the same access pattern alone: a coalesced index stream and one
        # scattered 4-byte read per index in a table of the mailbox's size
        ceil = ip.measure_gather(V * 4, 4, 1 << 28, 5)
        rate = edges_per_launch / (avg_ms * 1e-3)
        roofline["gather_ceiling"] = {
            "pattern": f"u32 index stream + one scattered 4-byte read per index, table {V * 4 >> 20} MiB "
                       "(the 4-byte mailbox), ipg_measure_gather",
            "rows_per_s": round(ceil["rows_per_s"] / 1e9, 2), "kernel_edges_per_s": round(rate / 1e9, 2),
            "unit": "G/s", "frac": round(rate / ceil["rows_per_s"], 4) if ceil["rows_per_s"] else None}
    roofline.update(stored_traffic(top_name, bytes_per_launch))

    # ---- the same work as the reference arm: CC + hop-count SSSP ----
    same_work, res_hop, counts_hop = same_work_row(args, cc, g, E, world, barrier, max_over_ranks)

    # ---- end to end through the C ABI with host buffers ----
    e2e = None
    cc_labels_components = int(len(np.unique(res_cc)))
    reached = int(np.count_nonzero(res_sp != 0xFFFFFFFF))
    h_idx, h_adj, h_wgt = g.to_host()  # also the oracle's input for the parity checks
    if not args.no_e2e:
        idx, adj, wgt = h_idx, h_adj, h_wgt
        p_idx = ip.PinnedArray(V, np.uint64)
        p_adj = ip.PinnedArray(E, np.uint32)
        p_wgt = ip.PinnedArray(E, np.uint32)
        p_idx.array[:] = idx
        p_adj.array[:] = adj
        p_wgt.array[:] = wgt
        out_cc = ip.PinnedArray(V, np.uint32)
        out_sp = ip.PinnedArray(V, np.uint32)
        del idx, adj, wgt

        # Two resident graphs, allocated once.  Every step copies its inputs
        # into one of them (ipg_graph_refill_host: its own stream, no
        # allocation, no device-wide synchronisation), attaches and runs both
        # programs and reads both results back.  Sequential: copy, then
        # compute.  Pipelined: the copy of step k+1 runs on a second host
        # thread while step k computes on the other graph.
        gbuf = [ip.Graph.from_csr(V, E, p_idx.array, p_adj.array, wgt=p_wgt.array) for _ in range(2)]
        # The engines alternate between the two graphs, and a captured loop is
        # captured anew for every attached graph (about 10 ms a step here),
        # so these steps run the host-driven superstep loop.
        for eng in (cc, sp):
            eng.set_graph_loop(False)

        def refill(gr, err):
            try:
                gr.refill(p_idx.array, p_adj.array, p_wgt.array)
            except Exception as ex:  # re-raised by the step that needs the graph
                err.append(ex)

        def compute(gr):
            gr.set_symmetric(True)  # the workload is undirected: every edge has its reverse, same weight
            cc.attach(gr)
            cc.run_only()
            cc.values(out_cc.array)
            sp.attach(gr)
            sp.run_only()
            sp.values(out_sp.array)

        def e2e_sequential(nsteps):
            for _ in range(nsteps):
                err = []
                refill(gbuf[0], err)
                if err:
                    raise err[0]
                compute(gbuf[0])

        def e2e_pipelined(nsteps):
            err = []
            th = threading.Thread(target=refill, args=(gbuf[0], err))
            th.start()
            for k in range(nsteps):
                th.join()
                if err:
                    raise err[0]
                if k + 1 < nsteps:
                    th = threading.Thread(target=refill, args=(gbuf[(k + 1) % 2], err))
                    th.start()
                compute(gbuf[k % 2])

        def timed(run):
            run(2)  # both graphs' refill buffers made, engines attached once
            barrier()
            t0.record()
            run(args.steps)
            t1.record()
            barrier()
            return max_over_ranks(t0.elapsed_time(t1))

        ms_seq = timed(e2e_sequential)
        ms_e2e = timed(e2e_pipelined)
        e2e = {"value": round(replica_gteps(world, E, runs, ms_e2e), 4), "unit": "GTEPS",
               "h2d_bytes_per_step": int(V * 8 + E * 4 + E * 4), "d2h_bytes_per_step": int(2 * V * 4),
               "ms_per_step": round(ms_e2e / args.steps, 3),
               "path": "per step: ipg_graph_refill_host from pinned host CSR + weights into one of two resident "
                       "graphs, attach and run CC and SSSP (host-driven superstep loop), both results to pinned "
                       "host buffers; the next step's refill runs on a second host thread and stream while this "
                       "step computes",
               "sequential": {"value": round(replica_gteps(world, E, runs, ms_seq), 4),
                              "ms_per_step": round(ms_seq / args.steps, 3),
                              "path": "the same steps with no overlap: refill, then compute"}}
        e2e["results_equal_resident"] = bool(np.array_equal(out_cc.array, res_cc) and
                                             np.array_equal(out_sp.array, res_sp))
        for gr in gbuf:
            gr.free()
        for a in (p_idx, p_adj, p_wgt, out_cc, out_sp):
            a.free()
    cc.release()
    sp.release()

    # ---- CPU baseline: the reference's binaries on the same graph ----
    cpu, ref_dumps = None, {}
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu, ref_dumps = cpu_baseline_leg(g, E)
    g.free()

    # ---- parity of the timed runs' results (outside every timed region) ----
    parity = None
    if rank == 0 and not args.no_parity:
        parity = parity_check(V, E, h_idx, h_adj, h_wgt, res_cc, counts_cc, res_sp, res_hop, counts_hop, ref_dumps)
    del h_idx, h_adj, h_wgt

    # ---- the other workloads (one GPU only; each frees what it held) ----
    extra = {}
    if world == 1 and not args.no_extra:
        rows = (("pagerank_precision_split", lambda: pagerank_row(peak, not args.no_parity)),
                ("batched_many_graph", batch_row),
                ("serving", serving_row))
        wanted = set(args.rows.split(",")) if args.rows else None
        for name, fn in rows:
            if wanted is not None and name not in wanted:
                continue
            try:
                extra[name] = fn()
            except Exception as exc:  # report, keep the headline
                extra[name] = {"error": f"{type(exc).__name__}: {exc}"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": round(value, 4), "unit": "GTEPS", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 3), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": "synthetic",
            "config": {"workload": f"cc (spread) + weighted sssp from 0 (spread, atomicMin), undirected R-MAT "
                                   f"scale {scale}, edge factor 16, a/b/c=0.57/0.19/0.19, seed 1, weights U[1,255]",
                       "scale": scale, "vertices": V, "edges_stored": E, "parallelism": f"replicas x{world}",
                       "superstep_loop": "captured CUDA graph with a device-evaluated while condition",
                       "vertex_order": ("degree-ordered copy of the graph, built at the first attach (outside the "
                                        "timed region; e2e rebuilds it every step); results in the graph's own ids"
                                        if renamed else "the graph's own numbering"),
                       "teps": "Graph500: stored edges x runs / time",
                       "l2": "inputs (3.8 GB) larger than L2; no flush",
                       "traversed_gteps": round(traversed_gteps, 4),
                       "supersteps_cc_sssp": list(supersteps[0]) if supersteps else None,
                       "cc_components": cc_labels_components, "sssp_reached": reached},
            "parity": parity["ok"] if parity else None,
            "parity_detail": parity,
            "same_work_as_reference": same_work,
            "roofline": roofline,
            "cpu_baseline": cpu,
            "e2e": e2e,
            "gpu_launches": launches,
            "clocks": clk,
            "kernels": {k: {"launches": v["launches"], "ms": round(v["ms"], 3), "bytes": round(v["bytes"]),
                            "gbs": round(v["bytes"] / (v["ms"] * 1e-3) / 1e9, 1) if v["ms"] else None}
                        for k, v in sorted(prof.items(), key=lambda kv: -kv[1]["ms"])},
        }
        line.update(extra)
        print(json.dumps(line))
    if world > 1:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
