#!/usr/bin/env python
"""Benchmark: PHOLD committed events/s on the 65,536-LP ring workload (local array queue).

The local array queue runs in the form the shipped tuned shape names: the bucketed form
(per-LP time buckets of 8-byte keys, laq_mode 2) on the B200; `--laq-mode 0` selects the
sorted form (per-LP sorted rings, children merged every window).

Workload (synthetic, seeded): 65,536 LPs x 64 initial events, lookahead 0.1 + Exp(1)
float32 increments, 90% of destinations uniform within +-16 ring neighbours (self
excluded) and 10% uniform, end time 1000.0, per-LP capacity 256, seed 7.
One bench step = one complete run of that workload: populate the queues on the device,
then drain safe windows until the minimum timestamp reaches the end time.

  value  committed events / device time of the runs (CUDA events on the launching
         stream, inputs already resident in HBM; the queue arrays exceed L2: 1.07 GB
         of buckets in the bucketed form, 268 MB of rings in the sorted form)
  e2e    the same through the public C ABI with host buffers: per step the initial
         events are copied from page-locked host memory, and the per-LP results
         (count, checksum, order hash) are copied back

`--impl reference` times the CPU port of the reference's window loop (per-LP
std::priority_queue, all host threads) on a bounded sample of the same workload.

Multi-GPU (torchrun): every rank runs its own replica (seed + rank); value = events
of all ranks / max over ranks of the device time.
"""
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

WORKLOAD = dict(num_lps=65536, events_per_lp=64, lookahead=0.1, end_time=1000.0, seed=7, dest_mode=1,
                ring_width=16, ring_frac=0.9)
WORKLOAD_NAME = "phold_large_65536lp_x64_ring16_T1000"
METRIC = "PHOLD committed events/s"
UNIT = "events/s"
# Algorithmic bytes: 48 B per committed event (16 B item read, 16 B child write, 16 B
# per-LP state read-modify-write) + 4 B per LP per window (window minimum).
BYTES_PER_EVENT = 48
BYTES_PER_LP_WINDOW = 4


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi samples of SM clock and throttle reasons during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for ln in self.proc.stdout:
            self.lines.append(ln.strip())

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
        for ln in self.lines:
            parts = [x.strip() for x in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for nm, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def cpu_model():
    """The host CPU's model name (lscpu / /proc/cpuinfo)."""
    try:
        with open("/proc/cpuinfo") as fh:
            for ln in fh:
                if ln.lower().startswith("model name"):
                    return ln.split(":", 1)[1].strip()
    except Exception:
        pass
    return None


def golden(name):
    """Oracle results committed by tests/golden/make_phold_golden.py (None if absent)."""
    try:
        with open(os.path.join(ROOT, "tests", "golden", "phold_golden.json")) as fh:
            return json.load(fh).get(name)
    except Exception:
        return None


def matches_golden(O, g, r, s):
    """A run's result and per-LP outputs equal the committed oracle results, bit for bit."""
    return (g is not None and r["committed"] == g["committed"] and r["steps"] == g["windows"]
            and r["pending"] == g["pending"] and r["pending_csum"] == int(g["pending_csum"])
            and r["digest"] == int(g["digest"])
            and O.lp_sha256(s["count"], s["csum"], s["ohash"]) == g["lp_sha256"])


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def reduce_over_ranks(dist, x, op, device):
    """One float reduced over all ranks (op "max" or "sum"); x itself without a group."""
    if dist is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX if op == "max" else dist.ReduceOp.SUM)
    return float(t.item())


def replica_seed(rank):
    """Replica r of the multi-GPU bench runs the workload with seed + r."""
    return WORKLOAD["seed"] + rank


def cpu_reference_run(cfgd, end_time, threads):
    from oracle import oracle as O
    c = O.make_cfg(num_lps=cfgd["num_lps"], events_per_lp=cfgd["events_per_lp"], lookahead=cfgd["lookahead"],
                   end_time=end_time, seed=cfgd["seed"], dest_mode=cfgd["dest_mode"],
                   ring_width=cfgd["ring_width"], ring_frac=cfgd["ring_frac"])
    return O.phold(c, threads)


CPU_SAMPLE_END = 12.0  # bounded sample: the first 12 of 1000 time units (~45 M events)
CPU_SAMPLE_END_1T = 0.6  # the single-thread sample (~2.3 M events; one global 4.2 M-item heap)


def run_reference(args):
    ws, rank, _ = dist_env()
    if rank != 0:
        return 0
    threads = os.cpu_count() or 1
    vals = []
    committed = 0
    for i in range(args.warmup + args.steps):
        r = cpu_reference_run(WORKLOAD, CPU_SAMPLE_END, threads)
        if i >= args.warmup:
            vals.append(r["committed"] / r["seconds"])
            committed = r["committed"]
    v = statistics.median(vals)
    sample = (f"end_time {CPU_SAMPLE_END} of {WORKLOAD['end_time']} ({committed} events), same LPs/population/seed; "
              f"window-synchronous per-LP std::priority_queue port of the reference loop on {threads} threads")
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * committed / v, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD_NAME, "queue": "per-LP std::priority_queue (CPU)", "sample_end_time": CPU_SAMPLE_END},
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample,
                         "cpu_model": cpu_model()},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    return 0


# ---- the other forms of the hot path (rank 0, one GPU) ----

ASTAR_BYTES_PER_EXPANSION = {4: 17 + 5 * 4 + 20, 8: 17 + 5 * 8 + 20}  # pop + closed mark + neighbours + push


def _timed(fn, warmup, steps):
    for _ in range(warmup):
        fn()
    t0 = time.perf_counter()
    out = [fn() for _ in range(steps)]
    return out, time.perf_counter() - t0


def _astar_shape(grids, args, default, space=None):
    """The A* configuration for a bench batch: the tuner's (shipped or cached, timed when
    neither has the workload class) unless --no-tune."""
    if args.no_tune:
        return dict(default)
    from gpupq_b200 import autotune
    return autotune.tune_astar(grids, space=space, force=args.retune)


def bench_astar_plain(G, O, args, peak):
    """One 2048 x 2048 grid (Bernoulli(0.2), seed 3, corner to corner, 4-connected, 1024
    shards of 64 x 64): expansions (cells with f <= C*) per second of device time."""
    g = G.astar_grid(2048, 2048, 0.2, 3)
    shape = _astar_shape(g, args, dict(tile=64), space={"tile": [64]})  # 1024 shards, as the workload names
    with G.AStar(**shape) as a:
        def step():
            r = a.solve(g)
            return r[0], a.stats()
        out, wall = _timed(step, args.warmup, args.steps)
    exp = int(out[0][0]["expanded"])
    dev_s = sum(st["total_ms"] for _, st in out) / 1e3
    want = O.astar({k: int(g[0][k]) for k in O.ASTAR_FIELDS})
    exact = all(int(r[k]) == want[k] for r, _ in out for k in ("cost", "expanded", "gsum", "path_len", "path_hash"))
    achieved = exp * ASTAR_BYTES_PER_EXPANSION[4] * args.steps / dev_s / 1e9
    return {"workload": "astar_plain_2048x2048_p0.2_4conn_1024shards", "metric": "A* expansions/s",
            "value": exp * args.steps / dev_s, "unit": "expansions/s", "cost": int(out[0][0]["cost"]),
            "expanded": exp, "ms_per_query": 1e3 * dev_s / args.steps, "exact_vs_oracle": exact, "config": shape,
            "e2e": {"value": exp * args.steps / wall, "unit": "expansions/s", "h2d_bytes_per_step": 32,
                    "d2h_bytes_per_step": 48},
            "roofline": {"bound": "latency (critical path of ~4100 dependent expansions)", "achieved": achieved,
                         "peak": peak, "unit": "GB/s", "frac": achieved / peak},
            "cpu_baseline": {"value": want["expanded"] / want["seconds"], "unit": "expansions/s", "cores": 1,
                             "kind": "port", "sample": "the whole query, sequential std::priority_queue A*",
                             "cpu_model": cpu_model()}}


def bench_astar_batched(G, O, args, peak):
    """10,000 queries in one persistent launch: side log-uniform in [64, 1024], density
    uniform in [0.1, 0.3], 8-connected 10/14, octile, seeds 11 + i."""
    q = G.astar_queries(11, 10000, 8, 64, 1024, 0.1, 0.3)
    shape = _astar_shape(q, args, dict(tile=64, window=100))
    with G.AStar(**shape) as a:
        def step():
            r = a.solve(q)
            return r, a.stats()
        out, wall = _timed(step, args.warmup, args.steps)
        exp = int(out[0][0]["expanded"].sum())
        dev_s = sum(st["total_ms"] for _, st in out) / 1e3
        # the plain form: one launch per query, on the first 200
        pe, pt = 0, 0.0
        for i in range(200):
            r = a.solve(q[i:i + 1])
            pe += int(r[0]["expanded"])
            pt += a.stats()["total_ms"] / 1e3
    # every query against the sequential oracle (all host threads, outside the timing)
    allq = [{k: int(q[i][k]) for k in O.ASTAR_FIELDS} for i in range(len(q))]
    threads = os.cpu_count() or 1
    sec_all, res_all = O.astar_batch(allq, threads)
    fields = ("cost", "expanded", "gsum", "path_len", "path_hash")
    mism = [i for i in range(len(q)) for k in fields if int(out[0][0][i][k]) != res_all[i][k]]
    exact = all(int(out[j][0][i][k]) == int(out[0][0][i][k]) for j in range(len(out)) for i in range(len(q))
                for k in fields) and not mism
    sec, res = O.astar_batch(allq[:300], threads)
    achieved = exp * ASTAR_BYTES_PER_EXPANSION[8] * args.steps / dev_s / 1e9
    return {"workload": "astar_batched_10000q_side64-1024_8conn", "metric": "A* expansions/s (batched)",
            "value": exp * args.steps / dev_s, "unit": "expansions/s", "queries": len(q),
            "ms_per_batch": 1e3 * dev_s / args.steps, "bad_status": int((out[0][0]["status"] != 0).sum()),
            "config": shape,
            "plain_value": pe / pt, "plain_sample": "first 200 queries, one launch each",
            "batched_over_plain": (exp * args.steps / dev_s) / (pe / pt), "exact_vs_oracle": exact,
            "exact_checked": f"all {len(q)} queries of every timed batch against the sequential oracle "
                             f"({sec_all:.1f} s on {threads} host threads); mismatches {len(set(mism))}",
            "e2e": {"value": exp * args.steps / wall, "unit": "expansions/s",
                    "h2d_bytes_per_step": int(q.nbytes), "d2h_bytes_per_step": int(len(q) * 48)},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak},
            "cpu_baseline": {"value": sum(r["expanded"] for r in res) / sec, "unit": "expansions/s", "cores": threads,
                             "kind": "port", "sample": "first 300 queries, one sequential A* per host thread",
                             "cpu_model": cpu_model()}}


C1 = dict(num_lps=1024, events_per_lp=16, lookahead=1.0, end_time=100.0, seed=42, dest_mode=0)


def _phold_form(G, O, cfgd, queue, runs, warmup=1, **kw):
    """Device-timed whole runs of one queue kind; (events/s, ms per run, windows, result,
    per-LP stats of the first timed run)."""
    cfg = G.make_phold_config(**cfgd, queue=queue, **kw)
    with G.Phold(cfg) as h:
        for _ in range(warmup):
            h.populate()
            h.run()
        ev, ms, first = 0, 0.0, None
        for _ in range(runs):
            h.populate()
            h.run()
            r = h.result()
            if first is None:
                first = (r, h.lp_stats())
            ev += r["committed"]
            ms += r["elapsed_ms"]
    return ev / (ms / 1e3), ms / runs, first


def bench_phold_c1(G, O, args, peak):
    """1,024 LPs x 16 events, lookahead 1.0 + Exp(1), uniform destinations, end time 100,
    seed 42 (820,705 events in 100 windows), through the parallel heap queue -- the kind
    the workload names, in its whole-GPU form and its one-CTA form -- with the four other
    kinds beside it; each checked against the committed oracle results, bit for bit."""
    g = golden("phold_plain_1024lp_x16_T100")
    kinds = {}
    # "hq": the default node size (the reference's 256 K root, here lowered to the
    # 16,384-item population: one node, worked by the whole GPU); "hq_one_cta": 1,024-item
    # nodes, one CTA working the heap
    for label, queue, kw in (("hq", "hq", {}), ("hq_one_cta", "hq", {"node_size": 1024}), ("laq", "laq", {}),
                             ("lhq", "lhq", {}), ("lsq", "lsq", {}), ("gaq", "gaq", {}),
                             ("gaq_graph", "gaq", {"gaq_engine": 1})):
        v, ms, (r, st) = _phold_form(G, O, C1, queue, runs=3, **kw)
        by = BYTES_PER_EVENT * r["committed"] + BYTES_PER_LP_WINDOW * C1["num_lps"] * r["steps"]
        kinds[label] = {"value": v, "ms_per_run": ms, "exact_vs_oracle": matches_golden(O, g, r, st),
                        "roofline_frac": by / (ms / 1e3) / 1e9 / peak}
    cpu = []
    for _ in range(5):  # one thread, median of 5 (the sequential oracle, the whole run)
        o = O.phold(O.make_cfg(**C1), 0)
        cpu.append(o["committed"] / o["seconds"])
    hq = kinds["hq"]
    achieved = hq["roofline_frac"] * peak
    return {"workload": "phold_plain_1024lp_x16_T100_heap_queue", "metric": "PHOLD committed events/s",
            "value": hq["value"], "unit": "events/s", "events_per_run": g["committed"] if g else None,
            "windows_per_run": g["windows"] if g else None, "exact_vs_oracle": hq["exact_vs_oracle"],
            "kinds": kinds, "timing": "device time of whole runs (CUDA events), 3 runs after 1 warm-up",
            "roofline": {"bound": "latency (0.3 MB working set, L2-resident)", "achieved": achieved, "peak": peak,
                         "unit": "GB/s", "frac": hq["roofline_frac"]},
            "cpu_baseline": {"value": statistics.median(cpu), "unit": "events/s", "cores": 1, "kind": "port",
                             "sample": "the whole run, sequential std::priority_queue oracle, median of 5",
                             "cpu_model": cpu_model()}}


def bench_phold_c2_gaq(G, O, args, peak):
    """The 65,536-LP ring workload to end time 1000 through the global array queue (one
    sorted array for all LPs; each window's children sorted and merged in), checked against
    the committed oracle results: as one sorted array worked by the whole GPU in one
    cooperative launch (the default), and as the per-window kernel sequence (radix sort,
    merge) replayed as a CUDA graph."""
    name = "phold_large_65536lp_x64_ring16_T1000"
    g = golden(name)
    cfgd = {k: WORKLOAD[k] for k in ("num_lps", "events_per_lp", "lookahead", "end_time", "seed", "dest_mode",
                                     "ring_width")}
    forms = {}
    for label, eng in (("one_launch", 0), ("graph", 1)):
        v, ms, (r, st) = _phold_form(G, O, cfgd, "gaq", runs=2, capacity=256, gaq_engine=eng)
        by = BYTES_PER_EVENT * r["committed"] + BYTES_PER_LP_WINDOW * cfgd["num_lps"] * r["steps"]
        forms[label] = {"value": v, "ms_per_run": ms, "windows_per_run": r["steps"],
                        "exact_vs_oracle": matches_golden(O, g, r, st), "achieved_gbs": by / (ms / 1e3) / 1e9}
    one = forms["one_launch"]
    return {"workload": name + "_global_array_queue", "metric": "PHOLD committed events/s", "value": one["value"],
            "unit": "events/s", "ms_per_run": one["ms_per_run"], "windows_per_run": one["windows_per_run"],
            "exact_vs_oracle": one["exact_vs_oracle"], "engines": forms,
            "timing": "device time of whole runs (CUDA events), 2 runs after 1 warm-up",
            "roofline": {"bound": "latency and grid barriers (three phases per window; the 4 M-item array "
                                  "is rewritten every window)",
                         "achieved": one["achieved_gbs"], "peak": peak, "unit": "GB/s",
                         "frac": one["achieved_gbs"] / peak}}


def bench_phold_long_queues(G, O, args, peak):
    """Long per-LP queues (what the reference's local array queue backed by a heap is for,
    src/local_array_queue.cu:517-561,603-681): 4,096 LPs with 4,096 pending events each,
    lookahead 0.01 (about 40 safe events per LP per window), ring +-16, end time 2 --
    through the bucketed local array queue (near events in time buckets, far ones in the
    per-LP spill lists), the sorted form and the per-LP heap; each checked against the
    committed oracle results."""
    name = "phold_long_4096lp_x4096_ring16_T2"
    g = golden(name)
    cfgd = dict(g["config"]) if g else dict(num_lps=4096, events_per_lp=4096, lookahead=0.01, end_time=2.0, seed=23,
                                            dest_mode=1, ring_width=16)
    forms = {}
    for label, queue, kw in (("laq_time_buckets", "laq", dict(laq_mode=2, capacity=8192)),
                             ("laq_sorted", "laq", dict(laq_mode=0, capacity=8192, insert_capacity=128)),
                             ("local_heap", "lhq", dict(capacity=8192, insert_capacity=128))):
        v, ms, (r, st) = _phold_form(G, O, cfgd, queue, runs=2, **kw)
        forms[label] = {"value": v, "ms_per_run": ms, "exact_vs_oracle": matches_golden(O, g, r, st)}
    best = forms["laq_time_buckets"]
    by = BYTES_PER_EVENT * (g["committed"] if g else 0) + BYTES_PER_LP_WINDOW * cfgd["num_lps"] * (
        g["windows"] if g else 0)
    achieved = by / (best["ms_per_run"] / 1e3) / 1e9
    return {"workload": name, "metric": "PHOLD committed events/s", "value": best["value"], "unit": "events/s",
            "exact_vs_oracle": best["exact_vs_oracle"], "forms": forms,
            "timing": "device time of whole runs (CUDA events), 2 runs after 1 warm-up",
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak}}


def bench_reference_own_queues(G, O, args, peak):
    """The reference's OWN local array, local heap and local splay queues with its DES
    loop (oracle/_ref, built from its unmodified sources by oracle/build_ref.py, the PHOLD
    adapter model one event per LP per window) on this GPU, beside this engine on the same
    workloads: the 1,024-LP workload and the 65,536-LP ring workload cut to end time 3.
    The reference's rate is its own figure (committed events over its simulation time,
    src/des.cu:95-122); every run is checked against the committed oracle results."""
    import subprocess
    import tempfile
    from oracle import build_ref as B
    golden_of = {"c1": "phold_plain_1024lp_x16_T100", "c2r": "phold_large_65536lp_x64_ring16_T3"}
    out = {}
    for variant, (queue, w) in B.VARIANTS.items():
        exe = B.binary_path(variant)
        g = golden(golden_of[w])
        entry = {"workload": golden_of[w]}
        if not os.path.exists(exe):
            entry["reference"] = "binary missing (python oracle/build_ref.py)"
            out[variant] = entry
            continue
        with tempfile.TemporaryDirectory() as td:
            res = os.path.join(td, "r.bin")
            p = subprocess.run([exe, res], capture_output=True, text=True, timeout=600)
            ok = p.returncode == 0
            eps = None
            for ln in p.stdout.splitlines():
                if ln.strip().startswith("Events per sec.:"):
                    eps = float(ln.split(":")[1].split("=")[0])
            if ok:
                raw = open(res, "rb").read()
                hdr = np.frombuffer(raw[:64], np.uint64)
                L = int(hdr[0])
                cnt = np.frombuffer(raw[64:64 + 4 * L], np.uint32)
                cs = np.frombuffer(raw[64 + 4 * L:64 + 12 * L], np.uint64)
                oh = np.frombuffer(raw[64 + 12 * L:64 + 20 * L], np.uint64)
                entry["reference_exact_vs_oracle"] = bool(g and O.lp_sha256(cnt, cs, oh) == g["lp_sha256"]
                                                          and int(hdr[1]) == g["committed"])
                entry["reference_windows"] = int(hdr[2])
        entry["reference_events_per_s"] = eps
        cfgd = dict(g["config"])
        kw = {"laq": dict(laq_mode=2 if w == "c2r" else 0), "lhq": {}, "lsq": {}}[queue]
        v, ms, (r, st) = _phold_form(G, O, cfgd, queue, runs=3, **kw)
        entry["ours_events_per_s"] = v
        entry["ours_exact_vs_oracle"] = matches_golden(O, g, r, st)
        entry["ours_over_reference"] = (v / eps) if eps else None
        out[variant] = entry
    best = max((e.get("ours_over_reference") or 0) for e in out.values())
    return {"metric": "PHOLD committed events/s, the reference's own queues vs this engine (same GPU)",
            "unit": "events/s", "variants": out, "max_ours_over_reference": best,
            "note": "reference timing includes its per-window host round trips (src/des.cu:179-214); ours is "
                    "device time of the persistent launch"}


ASTAR_REF_BYTES_PER_POP = 16 + 8 * 3 + 3 * 18  # pop + 8 neighbours (wall/closed bits, f_ol) + ~3 pushes with f_ol


def bench_astar_ref(G, O, args, peak):
    """The reference's own A* agent model (half-precision f, eight pops per round, stop at
    the goal) at its preset's shape: one 256 x 256 map with obstacle squares (0.2 of the
    cells, mean side 1), 2,048 concurrent agent slots, a pool of 16,384 agents; agents/s.
    Every agent is checked against the CPU oracle of the same semantics."""
    m = G.astar_ref_map(256, 256, 0.2, 1.0, seed=14580)
    agents = G.astar_ref_agents(m, 16384, seed=11)
    with G.AStarRef(256, 256, slots=2048) as a:
        for _ in range(2):
            r = a.solve(m, agents)
        ms, walls = [], []
        for _ in range(max(3, args.steps)):
            t0 = time.perf_counter()
            r2 = a.solve(m, agents)
            walls.append(time.perf_counter() - t0)
            ms.append(a.last_ms())
            same = all(np.array_equal(r2[k], r[k]) for k in ("found", "pops", "rounds", "cost"))
            if not same:
                raise SystemExit("reference-semantics A* is not reproducible")
    dev_s = statistics.median(ms) / 1e3
    threads = os.cpu_count() or 1
    sec_all, want = O.astar_ref(m, agents, threads)
    exact = (all(np.array_equal(r[k], want[k]) for k in ("found", "pops", "rounds"))
             and np.array_equal(r["cost"].view(np.uint32), want["cost"].view(np.uint32)))
    pops = int(r["pops"].sum())
    sample = 2048
    sec, _ = O.astar_ref(m, agents[:sample], threads)
    achieved = pops * ASTAR_REF_BYTES_PER_POP / dev_s / 1e9
    return {"workload": "astar_reference_semantics_256x256_2048slots_16384agents",
            "metric": "A* agents/s (reference semantics)", "value": len(agents) / dev_s, "unit": "agents/s",
            "pops_per_s": pops / dev_s, "ms_per_pool": 1e3 * dev_s, "found": int(r["found"].sum()),
            "mean_pops_per_agent": pops / len(agents), "exact_vs_oracle": bool(exact),
            "exact_checked": f"all {len(agents)} agents (found, f at the goal, pops, rounds) against the CPU oracle",
            "e2e": {"value": len(agents) / statistics.median(walls), "unit": "agents/s",
                    "h2d_bytes_per_step": int(m.nbytes + agents.nbytes),
                    "d2h_bytes_per_step": int(len(agents) * G.ASTAR_REF_RESULT_DTYPE.itemsize)},
            "roofline": {"bound": "latency (dependent heap levels per warp; state L2-resident)", "achieved": achieved,
                         "peak": peak, "unit": "GB/s", "frac": achieved / peak},
            "cpu_baseline": {"value": sample / sec, "unit": "agents/s", "cores": threads, "kind": "port",
                             "sample": f"first {sample} agents, one sequential agent per host thread",
                             "cpu_model": cpu_model()},
            "reference_binary": "not run: its kernel calls __syncthreads() in a thread-dependent branch "
                                "(src/a_star.cu:526-554), undefined on sm_70 and later"}


def bench_phold_batched(G, O, args, peak):
    """The PHOLD runs of the first second of the served stream (LPs log-uniform in
    [256, 65536], 32 events per LP, lookahead 0.5, end time 200), all in one launch of a
    session whose LP space holds rings (the default session form); the same batch in
    a time-bucket session and the plain path (each run alone through its own handle, both
    queue forms) beside it."""
    reqs, n = G.serve_stream(99, 2000.0, 1.0)
    runs = [reqs[i].phold for i in range(n) if reqs[i].kind == G.REQ_PHOLD]
    lps = sum(r.num_lps for r in runs)

    def batch(bucketed, warmup, steps):
        with G.PholdSession(max_lps=lps, max_instances=len(runs), bucketed=bucketed) as s:
            def step():
                t0 = time.perf_counter()
                for r in runs:
                    s.admit(r)
                s.step(0)
                got = s.collect()
                return got, time.perf_counter() - t0
            out, _ = _timed(step, warmup, steps)
        return sum(r.committed for _, r in out[0][0]), sum(t for _, t in out), out[0][0]

    ev, dt, got = batch(False, args.warmup, args.steps)
    ev0, dt0, got0 = batch(True, 1, args.steps)
    same = sorted((r.committed, r.digest) for _, r in got) == sorted((r.committed, r.digest) for _, r in got0)
    # the plain path: each run alone through its own handle.  Handles are created before
    # the timing, as the batch's session is; each timed run is populate + all windows +
    # result, as each timed batch step is admit + all windows + collect.
    plain = {}
    for mode in (2, 0):
        pe, pt, pw = 0, 0.0, 0.0
        handles = [G.Phold(G.make_phold_config(r.num_lps, 32, 0.5, 200.0, r.seed, laq_mode=mode,
                                               **({"block_threads": 512} if mode == 2 else {})))
                   for r in runs[:16]]
        try:
            for h in handles:  # warm-up
                h.populate()
                h.run()
                h.result()
            for h in handles:
                t0 = time.perf_counter()
                h.populate()
                h.run()
                rr = h.result()
                pw += time.perf_counter() - t0
                pe += rr["committed"]
                pt += rr["elapsed_ms"] / 1e3
        finally:
            for h in handles:
                h.close()
        plain[mode] = (pe / pw, pe / pt)
    pv = max(plain[2][0], plain[0][0])
    pdv = max(plain[2][1], plain[0][1])
    achieved = ev * BYTES_PER_EVENT * args.steps / dt / 1e9
    return {"workload": f"phold_batched_{len(runs)}runs_lp256-65536_x32_T200", "metric": "PHOLD events/s (batched)",
            "value": ev * args.steps / dt, "unit": "events/s", "runs": len(runs), "lps": lps,
            "ms_per_batch": 1e3 * dt / args.steps, "queue_form": "rings",
            "time_bucket_session_value": ev0 * args.steps / dt0, "same_results_both_forms": same,
            "plain_value": pv, "plain_bucketed_value": plain[2][0], "plain_sorted_value": plain[0][0],
            "plain_device_value": pdv,
            "plain_sample": "first 16 runs, each alone through its own handle created before the timing "
                            "(populate + run + result on the host clock, like admit + step + collect of the "
                            "batch), bucketed and sorted queue forms; plain_value is the faster; "
                            "plain_device_value counts device time only",
            "batched_over_plain": (ev * args.steps / dt) / pv,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak},
            "timing": "host wall clock around admit + session step (populate, all windows) + collect"}


def bench_served(G, args, duration):
    """The mixed stream: Poisson 2000/s, 80% A* (4-connected, side log-uniform in [128,
    4096], p 0.2), 20% PHOLD (LPs log-uniform in [256, 65536], 32 ev/LP, T 200), a 120 GiB
    budget; continuous batching vs one request per launch."""
    reqs, n = G.serve_stream(99, 2000.0, duration)
    out, st = G.serve(reqs, n, mode=G.SERVE_BATCHED, realtime=True, budget=120 << 30, tile=64)
    bad = sum(1 for i in range(n) if out[i].status != 0)

    def same(a, b, i):
        if reqs[i].kind == G.REQ_ASTAR:
            return all(getattr(a[i].astar, k) == getattr(b[i].astar, k)
                       for k in ("cost", "path_len", "expanded", "gsum", "path_hash"))
        return all(getattr(a[i].phold, k) == getattr(b[i].phold, k)
                   for k in ("committed", "steps", "pending", "pending_csum", "digest"))

    # every request of the timed stream, alone through the plain path (one launch each)
    aout, _ = G.serve(reqs, n, mode=G.SERVE_PLAIN, realtime=False, tile=64)
    exact_all = all(same(out, aout, i) for i in range(n))
    m = min(n, 150)
    pout, pst = G.serve(reqs, m, mode=G.SERVE_PLAIN, realtime=True, tile=64)
    bout, bst = G.serve(reqs, m, mode=G.SERVE_BATCHED, realtime=True, budget=120 << 30, tile=64)
    # saturated: the same prefix with every request present at the start
    sout, sst = G.serve(reqs, m, mode=G.SERVE_PLAIN, realtime=False, tile=64)
    tout, tst = G.serve(reqs, m, mode=G.SERVE_BATCHED, realtime=False, budget=120 << 30, tile=64)
    exact = all(same(bout, pout, i) for i in range(m))
    # an offered rate this GPU holds: the same mix at 600 requests/s for 2 s
    hreqs, hn = G.serve_stream(99, 600.0, 2.0)
    hout, hst = G.serve(hreqs, hn, mode=G.SERVE_BATCHED, realtime=True, budget=120 << 30, tile=64)
    hbad = sum(1 for i in range(hn) if hout[i].status != 0)
    r = lambda d: {k: (round(v, 6) if isinstance(v, float) else v) for k, v in d.items()}
    return {"workload": f"served_poisson2000_{duration:g}s_80astar_20phold", "metric": "served queries/s",
            "value": st["throughput"], "unit": "queries/s", "requests": n, "bad_status": bad,
            "offered_rate": 2000.0, "batched": r(st),
            "sustained_offered_rate": False,
            "exact_mix_equals_alone": exact_all,
            "exact_scope": "every request of the timed stream against the same request alone (plain path)",
            "capacity_note": "the PHOLD share alone needs about 20 G events/s at 2,000 requests/s "
                             "(400 runs/s x ~11,800 LPs x 32 events x ~133 events per chain), above the "
                             "batched engine's ~17 G events/s: the offered rate is beyond one GPU",
            "held_rate": {"offered_rate": 600.0, "seconds": 2.0, "requests": hn, "bad_status": hbad,
                          "batched": r(hst),
                          "sustained": bool(hst["throughput"] >= 0.9 * hn / 2.0 and hst["p99"] < 0.5)},
            "prefix": {"requests": m, "batched": r(bst), "plain": r(pst),
                       "batched_over_plain_throughput": bst["throughput"] / pst["throughput"],
                       "saturated_batched": r(tst), "saturated_plain": r(sst),
                       "saturated_batched_over_plain_throughput": tst["throughput"] / sst["throughput"],
                       "exact_mix_equals_alone": exact},
            "latency_unit": "s (finished - arrival, host clock)"}


def run_case(name):
    """Small named workloads for profiling captures (each runs its kernel twice)."""
    import gpupq_b200 as G
    if name == "astar_batched_1000":
        q = G.astar_queries(11, 1000, 8, 64, 1024, 0.1, 0.3)
        with G.AStar(tile=64, window=100) as a:
            for _ in range(2):
                r = a.solve(q)
            print(a.stats(), int(r["expanded"].sum()), int(r["pops"].sum()), int((r["status"] != 0).sum()))
    elif name == "astar_plain_2048":
        # the bench line's tuned shape: 1,024 shards of 64 x 64, f-window 1, one CTA per SM
        g = G.astar_grid(2048, 2048, 0.2, 3)
        with G.AStar(tile=64, window=1, ctas_per_sm=1) as a:
            for _ in range(2):
                r = a.solve(g)
            print(a.stats(), int(r[0]["expanded"]))
    elif name == "gaq_sort_32m":
        # the global array queue's post of 32 Mi items: min/max, 4 radix passes, merge
        import time
        N, L = 32 << 20, 65536
        rng = np.random.default_rng(5)
        items = np.zeros(N, G.ITEM_DTYPE)
        items["ts"] = rng.uniform(0, 1000, N).astype(np.float32)
        items["lp"] = rng.integers(0, L, N, dtype=np.uint32)
        items["id"] = np.arange(N, dtype=np.uint32)
        for _ in range(2):
            with G.Queue("gaq", num_lps=L, capacity=N // L + 1, insert_capacity=N // L + 1) as q:
                q.insert(items)
                t = time.perf_counter()
                q.post()
                print(f"post of {N} items: {(time.perf_counter() - t) * 1e3:.2f} ms (host clock)")
    elif name == "phold_c1_heap":
        # C1 through the whole-GPU heap queue (one 16,384-item root), two runs
        cfg = G.make_phold_config(**C1, queue="hq")
        with G.Phold(cfg) as h:
            for _ in range(2):
                h.populate()
                h.run()
                r = h.result()
            print(r["committed"], r["steps"], r["elapsed_ms"], h.launch_info())
    elif name == "gaq_array_c2_t20":
        # the 65,536-LP ring workload to end time 20 through the global array queue as one
        # sorted array in one launch (76 M events, 200 windows), two runs
        cfgd = {k: WORKLOAD[k] for k in ("num_lps", "events_per_lp", "lookahead", "seed", "dest_mode", "ring_width")}
        cfg = G.make_phold_config(**cfgd, end_time=20.0, queue="gaq", capacity=256)
        with G.Phold(cfg) as h:
            for _ in range(2):
                h.populate()
                h.run()
                r = h.result()
            print(r["committed"], r["steps"], r["elapsed_ms"], h.launch_info())
    elif name == "astar_ref_2048":
        m = G.astar_ref_map(256, 256, 0.2, 1.0, seed=14580)
        agents = G.astar_ref_agents(m, 4096, seed=11)
        with G.AStarRef(256, 256, slots=2048) as a:
            for _ in range(2):
                r = a.solve(m, agents)
            print(a.last_ms(), int(r["pops"].sum()))
    elif name == "served_held_rates":
        # the served mix at offered rates one B200 holds, over longer streams
        import json
        for rate, secs in ((600.0, 30.0), (800.0, 20.0)):
            reqs, n = G.serve_stream(99, rate, secs)
            out, st = G.serve(reqs, n, mode=G.SERVE_BATCHED, realtime=True, budget=120 << 30, tile=64)
            bad = sum(1 for i in range(n) if out[i].status != 0)
            print(json.dumps({"offered_rate": rate, "seconds": secs, "requests": n, "bad_status": bad,
                              **{k: (round(v, 4) if isinstance(v, float) else v) for k, v in st.items()}}))
    elif name in ("phold_batched_36", "phold_batched_36_buckets"):
        # the PHOLD runs among the first 0.1 s of the served stream, in a sorted-ring session
        # or (..._buckets) in a time-bucket session
        reqs, n = G.serve_stream(99, 2000.0, 0.1)
        runs = [reqs[i].phold for i in range(n) if reqs[i].kind == G.REQ_PHOLD][:40]
        with G.PholdSession(max_lps=sum(r.num_lps for r in runs), max_instances=len(runs),
                            bucketed=name.endswith("_buckets")) as s:
            for _ in range(2):
                for r in runs:
                    s.admit(r)
                s.step(0)
                got = s.collect()
            print(len(got), sum(r.committed for _, r in got))
    else:
        raise SystemExit(f"unknown case {name}")
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--queue", default="laq")
    ap.add_argument("--loop", default="persistent", choices=["persistent", "plain"])
    ap.add_argument("--laq-mode", type=int, default=None, choices=[0, 1, 2],
                    help="local array queue form (default: the tuned shape's)")
    ap.add_argument("--end-time", type=float, default=None, help="override the workload end time (debug)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-tune", action="store_true", help="skip the autotuner (library defaults)")
    ap.add_argument("--retune", action="store_true", help="ignore the autotuner cache")
    ap.add_argument("--tune-windows", type=int, default=200)
    ap.add_argument("--no-forms", action="store_true", help="skip the A*, batched and served sections")
    ap.add_argument("--served-seconds", type=float, default=1.0, help="length of the served request stream")
    ap.add_argument("--case", default=None,
                    choices=["astar_batched_1000", "astar_plain_2048", "phold_batched_36", "phold_batched_36_buckets",
                             "gaq_sort_32m",
                             "astar_ref_2048", "phold_c1_heap", "gaq_array_c2_t20", "served_held_rates"],
                    help="run one small named workload twice and exit (profiling captures)")
    args = ap.parse_args()
    if args.case:
        return run_case(args.case)
    if args.warmup < 3:
        ap.error("--warmup must be >= 3")
    if args.impl == "reference":
        return run_reference(args)

    ws, rank, local = dist_env()
    dist = None
    if ws > 1:
        import datetime
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    else:
        os.environ.setdefault("CUDA_VISIBLE_DEVICES", os.environ.get("CUDA_VISIBLE_DEVICES", "0"))

    import gpupq_b200 as G

    cfgd = dict(WORKLOAD)
    if args.end_time is not None:
        cfgd["end_time"] = args.end_time
    cfgd["seed"] = replica_seed(rank)
    shape = {}
    if not args.no_tune:
        from gpupq_b200 import autotune
        shape = autotune.tune_phold(dict(cfgd, capacity=256), queue=args.queue, loop=args.loop,
                                    windows=args.tune_windows, force=args.retune)
    if args.laq_mode is not None:
        if shape.get("laq_mode", 0) != args.laq_mode:
            shape = {"laq_mode": args.laq_mode}
            if args.laq_mode == 0:
                shape.update(lanes_per_lp=8, block_threads=128, insert_capacity=32)
            else:
                shape.update(block_threads=256)
    laq_mode = shape.get("laq_mode", 0) if args.queue == "laq" else 0
    form = {0: "", 1: "s", 2: "b"}[laq_mode]
    cfg = G.make_phold_config(**cfgd, queue=args.queue, capacity=256, loop=args.loop,
                              **dict({"insert_capacity": 64}, **shape))
    h = G.Phold(cfg)

    def barrier():
        if dist is not None:
            import torch
            torch.cuda.synchronize()
            dist.barrier()

    def max_over_ranks(x):
        return reduce_over_ranks(dist, x, "max", "cuda")

    def sum_over_ranks(x):
        return reduce_over_ranks(dist, x, "sum", "cuda")

    # warm-up; the first run is checked against the committed oracle results when the
    # workload is the one they were made for (seed 7: rank 0)
    ref_digest = None
    exact_vs_oracle = None
    for i in range(args.warmup):
        h.populate()
        h.run()
        r = h.result()
        if r["status_code"] != 0:
            raise SystemExit(f"run failed: {r}")
        ref_digest = (r["digest"], r["committed"])
        if i == 0:
            g = golden(WORKLOAD_NAME)
            if g is not None and all(g["config"][k] == cfgd[k] for k in g["config"]):
                from oracle import oracle as O
                exact_vs_oracle = matches_golden(O, g, r, h.lp_stats())

    barrier()
    sampler = ClockSampler(local if ws > 1 else 0)
    sampler.start()
    t_wall0 = time.perf_counter()
    dev_ms = 0.0
    committed = 0
    windows = 0
    for _ in range(args.steps):
        h.populate()
        h.run()
        r = h.result()
        if r["status_code"] != 0 or (r["digest"], r["committed"]) != ref_digest:
            raise SystemExit(f"run failed or not reproducible: {r}")
        dev_ms += r["elapsed_ms"]
        committed += r["committed"]
        windows += r["steps"]
    barrier()
    t_wall = time.perf_counter() - t_wall0
    clocks = sampler.stop()
    info = h.launch_info()

    dev_ms_max = max_over_ranks(dev_ms)
    committed_all = sum_over_ranks(committed)
    value = committed_all / (dev_ms_max / 1e3)
    ms_per_step = dev_ms_max / args.steps

    # roofline of the dominant kernel (the persistent window loop = the whole run)
    peak, peak_kind = load_peaks()
    per_run_bytes = BYTES_PER_EVENT * (committed / args.steps) + BYTES_PER_LP_WINDOW * cfgd["num_lps"] * (windows / args.steps)
    achieved = per_run_bytes / (dev_ms / args.steps / 1e3) / 1e9
    traffic = None
    tp = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(tp):
        try:
            t = json.load(open(tp))
            key = f"{args.queue}{form}_{args.loop}"
            if key in t:
                traffic = t[key]["dram_bytes_per_event"] * committed / args.steps
        except Exception:
            traffic = None

    # end-to-end through the C ABI with host buffers
    e2e = None
    if not args.no_e2e:
        n = cfgd["num_lps"] * cfgd["events_per_lp"]
        pin_ev = G.PinnedArray(n, G.ITEM_DTYPE)
        pin_ev.array[:] = G.initial_events(cfg)
        pc = G.PinnedArray(cfgd["num_lps"], np.uint32)
        ps = G.PinnedArray(cfgd["num_lps"], np.uint64)
        po = G.PinnedArray(cfgd["num_lps"], np.uint64)
        h.populate(pin_ev.array)
        h.run()
        h.result()
        barrier()
        t0 = time.perf_counter()
        ecommitted = 0
        for _ in range(args.steps):
            h.populate(pin_ev.array)
            h.run()
            r = h.result()
            h.lp_stats_into(pc.array, ps.array, po.array)
            ecommitted += r["committed"]
            if (r["digest"], r["committed"]) != ref_digest:
                raise SystemExit("e2e run differs from the device-resident run")
        barrier()
        e_wall = max_over_ranks(time.perf_counter() - t0)
        e2e = {"value": sum_over_ranks(ecommitted) / e_wall, "unit": UNIT,
               "h2d_bytes_per_step": int(n * G.ITEM_DTYPE.itemsize),
               "d2h_bytes_per_step": int(cfgd["num_lps"] * (4 + 8 + 8) + 64)}
        for p in (pin_ev, pc, ps, po):
            p.free()

    cpu = None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        threads = os.cpu_count() or 1
        rr = cpu_reference_run(WORKLOAD, CPU_SAMPLE_END, threads)
        cpu = {"value": rr["committed"] / rr["seconds"], "unit": UNIT, "cores": threads, "kind": "port",
               "sample": f"end_time {CPU_SAMPLE_END} of 1000 ({rr['committed']} events); window-synchronous per-LP "
                         f"std::priority_queue port of the reference loop on {threads} threads; the live "
                         f"population is constant (every event makes one child), so the per-event cost of "
                         f"the sample stands for the whole run",
               "cpu_model": cpu_model()}
        # one thread, median of 5 runs of the sequential oracle on a shorter sample (the
        # protocol the published single-core baselines use)
        one = [cpu_reference_run(WORKLOAD, CPU_SAMPLE_END_1T, 0) for _ in range(5)]
        cpu["single_thread"] = {"value": statistics.median(o["committed"] / o["seconds"] for o in one),
                                "unit": UNIT, "cores": 1,
                                "sample": f"end_time {CPU_SAMPLE_END_1T} of 1000 ({one[0]['committed']} events), "
                                          f"sequential std::priority_queue oracle, median of 5"}

    h.close()
    forms = None
    if rank == 0 and not args.no_forms:
        from oracle import oracle as O
        peak, _ = load_peaks()
        forms = {"phold_c1": bench_phold_c1(G, O, args, peak),
                 "phold_c2_gaq": bench_phold_c2_gaq(G, O, args, peak),
                 "phold_long_queues": bench_phold_long_queues(G, O, args, peak),
                 "reference_own_queues": bench_reference_own_queues(G, O, args, peak),
                 "astar_plain": bench_astar_plain(G, O, args, peak),
                 "astar_batched": bench_astar_batched(G, O, args, peak),
                 "astar_reference_semantics": bench_astar_ref(G, O, args, peak),
                 "phold_batched": bench_phold_batched(G, O, args, peak),
                 "served": bench_served(G, args, args.served_seconds)}
        if cpu is not None:  # the global array queue form runs the headline's workload
            forms["phold_c2_gaq"]["cpu_baseline"] = dict(cpu, note="the same workload and CPU runs as the line's "
                                                                   "cpu_baseline")
    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": ms_per_step, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic",
            "config": {"workload": WORKLOAD_NAME, "queue": args.queue, "loop": args.loop,
                       "end_time": cfgd["end_time"], "events_per_run": committed / args.steps,
                       "windows_per_run": windows / args.steps,
                       "laq_form": {0: "sorted rings", 1: "selection", 2: "time buckets"}[laq_mode]
                       if args.queue == "laq" else None,
                       "l2": ("inputs larger than L2 (1.07 GB bucket array)" if laq_mode == 2
                              else "inputs larger than L2 (268 MB queue array)"),
                       "parallelism": f"replicas x{ws}" if ws > 1 else "1 GPU",
                       "launch_shape": dict(shape, block_threads=info["block"], grid=info["grid"])},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": traffic,
                         "peak_source": f"{peak_kind} hbm_gbs", "kernel": ("lab_" if laq_mode == 2 else "phold_laq_") + args.loop,
                         "algorithmic_bytes_per_run": per_run_bytes},
            "exact_vs_oracle": exact_vs_oracle,
            "cpu_baseline": cpu,
            "e2e": e2e,
            "gpu_launches": int(args.steps * info["launches_per_run"]),
            "clocks": clocks,
            "wall_s_timed": t_wall,
            "forms": forms,
        }
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
