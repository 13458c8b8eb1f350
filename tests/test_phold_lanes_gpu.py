"""PHOLD with the lanes per LP that the library chooses from the number of LPs: just at and
just above each bound of the rule, and windows from nearly empty to ones in which almost
every event is safe, against the oracle."""
import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(cfgd, queue, loop="persistent", **kw):
    o = O.phold(O.make_cfg(**cfgd), 8)
    with G.Phold(G.make_phold_config(**cfgd, queue=queue, loop=loop, **kw)) as h:
        h.populate()
        h.run()
        r, s = h.result(), h.lp_stats()
    assert r["status_code"] == 0
    for k in ("committed", "steps", "pending", "pending_csum"):
        assert r[k] == o[k], k
    for k in ("count", "csum", "ohash"):
        assert np.array_equal(s[k], o[k]), k


# one wave of 148 x 1,024 threads: 32, 16, 8, 4 lanes, then one
@pytest.mark.parametrize("lps", [1, 2, 4736, 4737, 9472, 9473, 18944, 18945, 37888, 37889])
def test_splay_lanes(gpu_lib, lps):
    _check(dict(num_lps=lps, events_per_lp=9, lookahead=0.4, end_time=4.0, seed=lps, dest_mode=0), "lsq")


@pytest.mark.parametrize("lps,per,la,end", [(40, 1, 0.01, 3.0), (5000, 100, 20.0, 60.0), (10000, 70, 0.02, 0.6),
                                            (700, 200, 3.0, 20.0)])
def test_splay_split(gpu_lib, lps, per, la, end):
    """The split at the window's end: empty, whole and partial trees."""
    for loop in ("persistent", "plain"):
        _check(dict(num_lps=lps, events_per_lp=per, lookahead=la, end_time=end, seed=3, dest_mode=1, ring_width=3),
               "lsq", loop=loop, capacity=512, insert_capacity=512)


@pytest.mark.parametrize("lps", [1, 2048, 2049, 4096, 4097, 14208, 14209, 48000, 48001])
def test_sorted_array_lanes(gpu_lib, lps):
    for loop in ("persistent", "plain"):
        _check(dict(num_lps=lps, events_per_lp=9, lookahead=0.4, end_time=4.0, seed=lps, dest_mode=0), "laq", loop=loop)


@pytest.mark.parametrize("lps", [2049, 3552, 3553, 7104, 7105, 14209, 21312, 21313])
@pytest.mark.parametrize("per", [5, 24])
def test_sorted_array_lanes_by_events(gpu_lib, lps, per):
    """1.4 and 6.9 events per LP and window, around the waves of 32, 16 and 8 lanes."""
    _check(dict(num_lps=lps, events_per_lp=per, lookahead=0.4, end_time=3.0, seed=lps, dest_mode=0), "laq")


@pytest.mark.parametrize("lps,per,la,end,ring", [
    (1, 1, 0.5, 30.0, 0), (40, 1, 0.01, 3.0, 1), (4096, 9, 0.4, 6.0, 0), (4097, 9, 0.4, 6.0, 0), (4500, 17, 0.8, 8.0, 0),
    (300, 9, 3.0, 30.0, 1),     # most of a heap safe in every window
    (200, 73, 0.3, 6.0, 1), (200, 74, 0.02, 1.0, 1), (150, 600, 0.01, 0.4, 1),  # full levels, one more, four levels
    (200, 150, 20.0, 60.0, 1),  # more safe items than the warp form takes: event by event
])
def test_local_heap_windows(gpu_lib, lps, per, la, end, ring):
    for loop in ("persistent", "plain"):
        _check(dict(num_lps=lps, events_per_lp=per, lookahead=la, end_time=end, seed=per + lps, dest_mode=ring,
                    ring_width=3), "lhq", loop=loop, capacity=2048 if per > 256 else 512, insert_capacity=512)


@pytest.mark.parametrize("queue", ["lhq", "lsq"])
def test_largest_ctas(gpu_lib, queue):
    """CTAs of 1,024 threads, which the register use has to allow."""
    for loop in ("persistent", "plain"):
        _check(dict(num_lps=900, events_per_lp=9, lookahead=0.4, end_time=4.0, seed=4, dest_mode=0), queue, loop=loop,
               block_threads=1024)


@pytest.mark.parametrize("ibc", [1024, 33])
def test_sorted_array_insert_capacity(gpu_lib, ibc):
    """32 lanes per LP with the largest insert buffers (fewer LPs a CTA) and an odd size."""
    _check(dict(num_lps=300, events_per_lp=20, lookahead=0.3, end_time=6.0, seed=8, dest_mode=1, ring_width=4), "laq",
           insert_capacity=ibc)


@pytest.mark.parametrize("queue", ["laq", "lsq", "lhq"])
def test_state_goes_between_lane_counts(gpu_lib, queue):
    """A run's snapshot fits a handle that asks for the former default lanes, and back."""
    cfgd = dict(num_lps=900, events_per_lp=12, lookahead=0.5, end_time=12.0, seed=6, dest_mode=0)
    o = O.phold(O.make_cfg(**cfgd), 8)
    default = G.make_phold_config(**cfgd, queue=queue)
    asked = G.make_phold_config(**cfgd, queue=queue, lanes_per_lp=1 if queue == "lsq" else 8)
    for a, b in ((default, asked), (asked, default)):
        with G.Phold(a) as x, G.Phold(b) as y:
            x.populate()
            x.step(9)
            y.restore(x.snapshot())
            y.run()
            r, s = y.result(), y.lp_stats()
        assert r["committed"] == o["committed"]
        assert np.array_equal(s["ohash"], o["ohash"])
