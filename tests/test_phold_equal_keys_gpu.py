"""PHOLD runs from a caller's population in which events share their (timestamp, id): two LPs
start with the same events, whose children then meet in one LP.  A window takes them both,
one after the other, against a sequential model of the run."""
import heapq

import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def _mix(z):
    z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & M64
    z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & M64
    return z ^ (z >> 31)


def _model(cfgd, initial):
    ocfg = O.make_cfg(**cfgd)
    L, end = cfgd["num_lps"], np.float32(cfgd["end_time"])
    count, csum, ohash = np.zeros(L, np.uint32), [0] * L, [0] * L
    heap = [(int(t.view(np.uint32)), int(i), int(lp)) for t, i, lp in zip(initial["ts"], initial["id"], initial["lp"])]
    heapq.heapify(heap)
    while heap and np.uint32(heap[0][0]).view(np.float32) < end:
        bits, ident, lp = heapq.heappop(heap)
        h = _mix((ident << 32) | bits)
        csum[lp] = (csum[lp] + h) & M64
        ohash[lp] = (ohash[lp] + _mix((h + int(count[lp]) * 0x9e3779b97f4a7c15) & M64)) & M64
        count[lp] += 1
        ts, to = O.child(ocfg, np.array([bits], np.uint32).view(np.float32), [lp], [ident])
        heapq.heappush(heap, (int(ts.view(np.uint32)[0]), ident, int(to[0])))
    return count, np.array(csum, np.uint64), np.array(ohash, np.uint64)


@pytest.mark.parametrize("lanes", [0, 8])
@pytest.mark.parametrize("lps,per,la", [(64, 8, 0.5), (10, 40, 1.0), (2, 16, 2.0)])
@pytest.mark.parametrize("queue", ["lhq", "lsq"])
def test_equal_keys_in_one_lp(gpu_lib, queue, lps, per, la, lanes):
    cfgd = dict(num_lps=lps, events_per_lp=per, lookahead=la, end_time=6.0, seed=11, dest_mode=0)
    cfg = G.make_phold_config(**cfgd, queue=queue, capacity=1024, insert_capacity=512, max_steps=200,
                              lanes_per_lp=lanes if queue == "lhq" else 0)
    initial = G.initial_events(cfg)
    pairs = initial.reshape(lps, per)
    for k in ("ts", "id"):
        pairs[k][1::2] = pairs[k][0::2]
    count, csum, ohash = _model(cfgd, initial)
    with G.Phold(cfg) as h:
        h.populate(initial)
        h.run()
        r, s = h.result(), h.lp_stats()
    assert r["status_code"] == 0 and r["pending"] == lps * per
    assert r["committed"] == int(count.sum())
    assert np.array_equal(s["count"], count)
    assert np.array_equal(s["csum"], csum) and np.array_equal(s["ohash"], ohash)
