"""The workloads this framework is timed on, each through its public entry points.

A case is a dict of plain values; its "path" says which entry point it goes through:

  queue      a queue object stepped from the host: a batch of items goes in, then the loop of
             a discrete-event program (minimum; dequeue below minimum + window; a smaller
             batch of later items), and what is left at the end
  phold      one PHOLD run through a handle that the program keeps: populate, run, result
             and per-LP statistics
  session    many PHOLD runs of mixed sizes resident in one session
  astar      a batch of grid searches (n = 1: one search from corner to corner, and its path;
             eight cells in from the corners, which are walled in themselves on one map in seven)
  astar_ref  a pool of agents of the reference-semantics search on one map

Every output is a whole number or a bit pattern that follows from the inputs alone (event
counts, digests, per-LP checksums, costs, dequeued items), so equality says all there is to
say and there is no value in 64 bits to be near to.  Left out of the outputs is only what
depends on the clock or the schedule: elapsed times and, of the grid search, the numbers of
pops and of windows.
"""
import math
import random

import numpy as np

import gpupq_b200 as G


def listed():
    return [
        # a small model stepped from the host: launches, host round trips and small copies
        dict(name="queue_laq_1k", path="queue", kind="laq", lps=1024, per_lp=8, windows=8),
        # a larger, odd-sized model through the global array: bulk sort, merge, safe prefix
        dict(name="queue_gaq_20k", path="queue", kind="gaq", lps=20011, per_lp=16, windows=4),
        # the 1,024-LP preset with the default queue (sorted local arrays)
        dict(name="phold_laq_1k", path="phold", queue="laq", laq_mode=0, lps=1024, per_lp=16, lookahead=1.0,
             end_time=100.0, ring=0),
        # the 65,536-LP preset with time buckets, the benchmark's form, over a part of its time span
        dict(name="phold_buckets_64k", path="phold", queue="laq", laq_mode=2, lps=65536, per_lp=64, lookahead=0.1,
             end_time=50.0, ring=1),
        # the 1,024-LP preset with the heap queue, the kind it is benchmarked with
        dict(name="phold_hq_1k", path="phold", queue="hq", laq_mode=0, lps=1024, per_lp=16, lookahead=1.0,
             end_time=100.0, ring=0),
        # the 65,536-LP preset with the global array queue
        dict(name="phold_gaq_64k", path="phold", queue="gaq", laq_mode=0, lps=65536, per_lp=64, lookahead=0.1,
             end_time=10.0, ring=1),
        # local heaps: longer queues, an odd number of LPs
        dict(name="phold_lhq_8k", path="phold", queue="lhq", laq_mode=0, lps=8191, per_lp=120, lookahead=0.1,
             end_time=10.0, ring=1),
        # the 1,024-LP preset with local splay trees
        dict(name="phold_lsq_1k", path="phold", queue="lsq", laq_mode=0, lps=1024, per_lp=16, lookahead=1.0,
             end_time=100.0, ring=0),
        # a batch of simulations of the served mix's sizes in one session (default form, sorted rings)
        dict(name="session_48", path="session", runs=48, lps_lo=256, lps_hi=65536, per_lp=32, lookahead=0.5,
             end_time=50.0),
        # the 2048 x 2048 search and its path, in its tuned shape
        dict(name="astar_2048", path="astar", n=1, lo=2048, hi=2048, dens_lo=0.2, dens_hi=0.2, conn=4),
        # a twentieth of the batched searches' workload, in its tuned shape
        dict(name="astar_500", path="astar", n=500, lo=64, hi=1024, dens_lo=0.1, dens_hi=0.3, conn=8),
        # the reference's agents on its preset's map
        dict(name="astar_ref_4k", path="astar_ref", side=256, agents=4096, slots=2048),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _phold_end(lps, per_lp, lookahead, per_queue):
    """An end time of at most 100, 500 windows, 40 M events and `per_queue` events per LP, in whole windows."""
    t = min(100.0, 500 * lookahead, min(4.0e7 / lps, per_queue) * (1 + lookahead) / per_lp)
    return lookahead * max(2, int(t / lookahead))


def draw(rng):
    path = rng.choice(["queue", "phold", "phold", "phold", "session", "astar", "astar", "astar_ref"])
    if path == "queue":
        return dict(path=path, kind=rng.choice(["laq", "gaq"]), lps=int(_log(rng, 200, 20011)),
                    per_lp=rng.randint(2, 16), windows=rng.randint(2, 8))
    if path == "phold":
        queue, mode = rng.choice([("laq", 0), ("laq", 2), ("hq", 0), ("gaq", 0), ("lhq", 0), ("lsq", 0)])
        lps, per_lp = int(_log(rng, 500, 65536)), rng.randint(8, 64)
        la = rng.choice([0.1, 0.25, 0.5, 1.0])
        return dict(path=path, queue=queue, laq_mode=mode, lps=lps, per_lp=per_lp, lookahead=la,
                    end_time=_phold_end(lps, per_lp, la, 1600 if queue == "lsq" else 10000),
                    ring=rng.randint(0, 1))
    if path == "session":
        return dict(path=path, runs=rng.randint(2, 48), lps_lo=256, lps_hi=int(_log(rng, 1024, 65536)), per_lp=32,
                    lookahead=0.5, end_time=rng.choice([10.0, 25.0, 50.0]))
    if path == "astar":
        conn = rng.choice([4, 8])
        if rng.random() < 0.5:
            side, dens = int(_log(rng, 64, 2048)), rng.uniform(0.1, 0.3)
            return dict(path=path, n=1, lo=side, hi=side, dens_lo=dens, dens_hi=dens, conn=conn)
        return dict(path=path, n=int(_log(rng, 2, 500)), lo=64, hi=int(_log(rng, 128, 1024)), dens_lo=0.1,
                    dens_hi=0.3, conn=conn)
    return dict(path=path, side=rng.randint(64, 256), agents=int(_log(rng, 64, 4096)), slots=2048)


def work(case):
    """Bytes that the algorithm moves: PHOLD 48 per event (item in, child out, per-LP state)
    and 4 per LP and window; a search (17 + 5 N) per expanded cell and 20 per push; an agent
    94 per pop; a queue item 16 in and 16 out."""
    path = case["path"]
    if path == "queue":
        n = case["lps"] * case["per_lp"]
        return {"bytes": 32.0 * (n + case["windows"] * (n // (2 * case["windows"]))), "flops": 0}
    if path in ("phold", "session"):
        lps = case["lps"] if path == "phold" else \
            case["runs"] * (case["lps_hi"] - case["lps_lo"]) / math.log(case["lps_hi"] / case["lps_lo"])
        events = lps * case["per_lp"] * case["end_time"] / (1 + case["lookahead"])
        return {"bytes": 48.0 * events + 4.0 * lps * case["end_time"] / case["lookahead"], "flops": 0}
    if path == "astar":
        # side log-uniform in [lo, hi]: the mean of its square; about half of a grid is expanded
        cells = case["lo"] ** 2 if case["lo"] == case["hi"] else \
            (case["hi"] ** 2 - case["lo"] ** 2) / (2 * math.log(case["hi"] / case["lo"]))
        share = 0.5 if case["n"] == 1 else 0.05
        return {"bytes": case["n"] * cells * share * (37.0 + 5 * case["conn"]), "flops": 0}
    return {"bytes": 94.0 * case["agents"] * 0.2 * case["side"] ** 2, "flops": 0}


def _items(rng, lps, n, base, first_id):
    items = np.zeros(n, G.ITEM_DTYPE)
    items["ts"] = np.float32(base) + rng.standard_exponential(n, dtype=np.float32)
    items["lp"] = rng.permutation(np.arange(n, dtype=np.uint32) % np.uint32(lps))
    items["id"] = first_id + np.arange(n, dtype=np.uint32)
    return items


def prepare(case, seed):
    path, seed = case["path"], 1 + int(seed) % (1 << 40)
    if path == "queue":
        windows, n = case["windows"], case["lps"] * case["per_lp"]
        rng = np.random.default_rng(seed)
        batches = [_items(rng, case["lps"], n, 0.0, 0)]
        for w in range(windows):
            m = n // (2 * windows)
            batches.append(_items(rng, case["lps"], m, 4.0 * (w + 1) / windows, n + w * m))
        return dict(case=case, batches=batches, queue=G.Queue(case["kind"], case["lps"], capacity=64, insert_capacity=64))
    if path == "phold":
        la = case["lookahead"]
        arrivals = case["per_lp"] * max(la / (1 + la), 1 - math.exp(-la))  # children per LP and window, mean
        kw = dict(block_threads=512) if case["laq_mode"] == 2 else {}
        cfg = G.make_phold_config(case["lps"], case["per_lp"], la, case["end_time"], seed,
                                  dest_mode=G.DEST_RING if case["ring"] else G.DEST_UNIFORM, queue=case["queue"],
                                  laq_mode=case["laq_mode"], capacity=256 if case["per_lp"] <= 64 else 512,
                                  insert_capacity=64 if arrivals < 20 else 128, **kw)
        return dict(case=case, handle=G.Phold(cfg))
    if path == "session":
        rng = random.Random(seed)
        runs = [G.make_phold_config(int(_log(rng, case["lps_lo"], case["lps_hi"])), case["per_lp"],
                                    case["lookahead"], case["end_time"], rng.getrandbits(40))
                for _ in range(case["runs"])]
        session = G.PholdSession(max_lps=sum(r.num_lps for r in runs), max_instances=len(runs))
        return dict(case=case, runs=runs, session=session)
    if path == "astar":
        solver = G.AStar(tile=64, window=1 if case["conn"] == 4 else 100)
        if case["n"] == 1:
            side = case["lo"]
            grids = G.astar_grid(side, side, case["dens_lo"], seed, conn=case["conn"], start=8 * side + 8,
                                 goal=(side - 9) * side + side - 9)
            return dict(case=case, grids=grids, solver=solver, path=np.zeros(16 * side, np.uint32))
        grids = G.astar_queries(1000 * seed, case["n"], case["conn"], case["lo"], case["hi"], case["dens_lo"],
                                case["dens_hi"])
        return dict(case=case, grids=grids, solver=solver)
    m = G.astar_ref_map(case["side"], case["side"], 0.2, 1.0, seed=seed)
    return dict(case=case, map=m, agents=G.astar_ref_agents(m, case["agents"], seed=seed + 1),
                solver=G.AStarRef(case["side"], case["side"], slots=case["slots"]))


def _run_queue(state):
    q, batches = state["queue"], state["batches"]
    windows = state["case"]["windows"]
    step = np.float32(4.0 / windows)
    out = []
    q.insert(batches[0])
    q.post_init()
    left = len(batches[0])
    for later in batches[1:]:
        q.pre()
        out.append(q.dequeue(float(np.float32(q.get_min()) + step), capacity=left))
        if len(later):
            q.insert(later)
        q.post()
        left += len(later) - len(out[-1])
    out.append(q.dequeue(math.inf, capacity=left))
    return np.concatenate(out).view(np.int32)


def run(state):
    path = state["case"]["path"]
    if path == "queue":
        return _run_queue(state)
    if path == "phold":
        h = state["handle"]
        h.populate()
        h.run()
        r, s = h.result(), h.lp_stats()
        out = {k: r[k] for k in ("committed", "steps", "pending", "status_code")}
        out["final_min"] = np.array([r["final_min"]], np.float32).view(np.int32)
        out.update({k: np.array([r[k]], np.uint64).view(np.int64) for k in ("pending_csum", "digest")})
        out.update(count=s["count"].view(np.int32), csum=s["csum"].view(np.int64), ohash=s["ohash"].view(np.int64))
        return out
    if path == "session":
        slots = [state["session"].admit(r) for r in state["runs"]]
        state["session"].step(0)
        got = dict(state["session"].collect())
        return {k: np.array([getattr(got[s], k) for s in slots], np.uint64).view(np.int64)
                for k in ("committed", "steps", "pending", "pending_csum", "digest")}
    if path == "astar":
        r = state["solver"].solve(state["grids"])
        out = {k: r[k].copy().view(np.int32) for k in ("cost", "path_len", "status")}
        out.update({k: r[k].copy().view(np.int64) for k in ("expanded", "gsum", "path_hash")})
        if state["case"]["n"] == 1:
            cells = state["solver"].path(0, capacity=len(state["path"]))
            state["path"][:len(cells)] = cells
            state["path"][len(cells):] = 0
            out["path"] = state["path"].view(np.int32)
        return out
    r = state["solver"].solve(state["map"], state["agents"])
    out = {k: r[k].copy().view(np.int32) for k in ("found", "pops", "rounds", "status")}
    out["cost"] = r["cost"].copy().view(np.int32)  # the bits of f at the goal
    return out
