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
