"""A session whose LPs hold events of equal (timestamp, id), here from a snapshot that was given
such events: each takes a place of its own in its LP's sequence, against a sequential model."""
import struct

import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O
from tests.test_phold_equal_keys_gpu import _model

RING_REGION = 9  # the regions before it: runs, minima, errors, in use, LP's run, count, two sums, control


def _ring_at(snap):
    b = snap.tobytes()
    at = 8 + 4 * 12
    at += 8 + struct.unpack_from("<Q", b, at)[0] + 4
    for _ in range(RING_REGION):
        at += 8 + struct.unpack_from("<Q", b, at)[0]
    return at + 8, struct.unpack_from("<Q", b, at)[0]


@pytest.mark.gpu
@pytest.mark.parametrize("lps,per,la,cap", [(64, 8, 0.5, 256), (10, 40, 1.0, 256), (2, 30, 2.0, 256), (4, 200, 2.0, 1024),
                                            (2, 900, 3.0, 2048)])  # lists, more than a list, more than the warp's space
def test_equal_keys_in_one_lp(gpu_lib, lps, per, la, cap):
    cfgd = dict(num_lps=lps, events_per_lp=per, lookahead=la, end_time=6.0, seed=13, dest_mode=0)
    kw = dict(max_lps=lps, max_instances=1, capacity=cap, insert_capacity=1000, lanes_per_lp=32)
    with G.PholdSession(**kw) as s:
        slot = s.admit(G.make_phold_config(**cfgd))
        snap = s.snapshot()  # populated, no window yet
        at, size = _ring_at(snap)
        assert size == lps * cap * 16
        ring = snap[at:at + size].view(G.ITEM_DTYPE).reshape(lps, cap)
        events = ring[:, :per]
        for k in ("ts", "id"):
            events[k][1::2] = events[k][0::2]
        if per >= 200:  # and within an LP
            for k in ("ts", "id"):
                events[k][:, 1::2] = events[k][:, 0::2]
        initial = events.reshape(-1).copy()
        s.restore(snap)
        s.step(0)
        got = dict(s.collect())[slot]
    count, csum, ohash = _model(cfgd, initial)
    assert got.status == 0 and got.pending == lps * per
    assert got.committed == int(count.sum())
    assert got.digest == O.digest(count, csum, ohash)
