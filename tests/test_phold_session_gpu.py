"""GPU tests of resident PHOLD runs (gpq_phold_session_*): every run of a batch or of a
stream with admissions between steps commits exactly what it commits alone on the
single-run engine (committed count, windows, digest over the per-LP outputs, pending
events, final minimum)."""
import random

import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu

KEYS = ("committed", "steps", "pending", "pending_csum", "digest", "final_min")


def _alone(cfg):
    c = G.make_phold_config(cfg.num_lps, cfg.events_per_lp, cfg.lookahead, cfg.end_time, cfg.seed,
                            dest_mode=cfg.dest_mode, ring_width=cfg.ring_width or 16, queue="laq",
                            capacity=256, insert_capacity=64, loop="persistent")
    c.ring_threshold = cfg.ring_threshold
    with G.Phold(c) as h:
        h.populate()
        h.run()
        return h.result()


def _runs(seed, n):
    rng = random.Random(seed)
    out = []
    for i in range(n):
        L = rng.choice([1, 3, 40, 256, 700, 3000])
        ring = L > 40 and rng.random() < 0.5
        out.append(G.make_phold_config(L, rng.choice([1, 4, 16, 32]), rng.choice([0.1, 0.5, 1.0]),
                                       rng.choice([0.0, 5.0, 20.0, 60.0]), 1000 + i,
                                       dest_mode=G.DEST_RING if ring else G.DEST_UNIFORM, ring_width=16))
    return out


def _d(r):
    return r if isinstance(r, dict) else r.as_dict()


def _same(a, b):
    a, b = _d(a), _d(b)
    for k in KEYS:
        assert a[k] == b[k], (k, a[k], b[k])
    assert a["status"] == 0 and b["status"] == 0


@pytest.mark.parametrize("bucketed", [False, True])
def test_batch_equals_alone(gpu_lib, bucketed):
    runs = _runs(1, 24)
    with G.PholdSession(max_lps=sum(c.num_lps for c in runs), max_instances=64, bucketed=bucketed) as s:
        slot_of = {s.admit(c): i for i, c in enumerate(runs)}
        s.step(0)
        got = {slot_of[sl]: r for sl, r in s.collect()}
        assert s.usage() == (0, 0)
    assert len(got) == len(runs)
    for i, c in enumerate(runs):
        _same(got[i], _alone(c))


@pytest.mark.parametrize("bucketed", [False, True])
@pytest.mark.parametrize("windows", [1, 5, 40])
def test_stream_equals_alone(gpu_lib, windows, bucketed):
    """Runs admitted while others are mid-run, into an LP space that holds only some of
    them at a time (LPs and slots of finished runs are reused)."""
    runs = _runs(2, 20)
    want = [_alone(c) for c in runs]
    got, slot_of, pending, refused = {}, {}, list(range(len(runs))), 0
    with G.PholdSession(max_lps=4000, max_instances=8, bucketed=bucketed) as s:
        for _ in range(100000):
            while pending:
                sl = s.admit(runs[pending[0]])
                if sl is None:
                    refused += 1
                    break
                slot_of[sl] = pending.pop(0)
            s.step(windows)
            for sl, r in s.collect():
                got[slot_of.pop(sl)] = r
            if not pending and not slot_of:
                break
    assert refused > 0 and len(got) == len(runs)
    for i in range(len(runs)):
        _same(got[i], want[i])


def _drive(s, runs, slot_of, pending, windows, got):
    """Admit, step and collect until every run has finished; returns the results by run."""
    for _ in range(100000):
        while pending:
            sl = s.admit(runs[pending[0]])
            if sl is None:
                break
            slot_of[sl] = pending.pop(0)
        s.step(windows)
        for sl, r in s.collect():
            got[slot_of.pop(sl)] = _d(r)
        if not pending and not slot_of:
            return got
    raise AssertionError("runs did not finish")


@pytest.mark.parametrize("bucketed", [False, True])
def test_session_snapshot_resumes_exactly(gpu_lib, bucketed):
    """Snapshot a session mid-stream (some runs mid-run, one admitted but not started,
    LP ranges reused), finish it; restore the snapshot into a fresh session and into one
    that already holds other runs, finish those: every run ends the same three times and
    as it ends alone."""
    runs = _runs(3, 14)
    kw = dict(max_lps=4000, max_instances=8, bucketed=bucketed)
    with G.PholdSession(**kw) as s:
        slot_of, pending, got = {}, list(range(len(runs))), {}
        for _ in range(3):  # a few steps, with collections that free slots and LPs
            while pending:
                sl = s.admit(runs[pending[0]])
                if sl is None:
                    break
                slot_of[sl] = pending.pop(0)
            s.step(4)
            for sl, r in s.collect():
                got[slot_of.pop(sl)] = _d(r)
        if pending:  # one run admitted but not started when the snapshot is taken
            sl = s.admit(runs[pending[0]])
            if sl is not None:
                slot_of[sl] = pending.pop(0)
        snap = s.snapshot()
        state = (dict(slot_of), list(pending), dict(got))
        first = _drive(s, runs, slot_of, pending, 4, got)
    for target_busy in (False, True):
        with G.PholdSession(**kw) as t:
            if target_busy:
                for c in _runs(9, 3):
                    t.admit(c)
                t.step(2)
            t.restore(snap)
            slot_of, pending, got = dict(state[0]), list(state[1]), dict(state[2])
            again = _drive(t, runs, slot_of, pending, 4, got)
            assert t.usage() == (0, 0)
        assert sorted(again) == sorted(first) == list(range(len(runs)))
        for i in range(len(runs)):
            _same(again[i], first[i])
    for i, c in enumerate(runs):
        _same(first[i], _alone(c))


def test_session_snapshot_rejects_other_parameters(gpu_lib):
    with G.PholdSession(max_lps=1000, max_instances=4) as s:
        s.admit(_runs(4, 1)[0])
        snap = s.snapshot()
    with G.PholdSession(max_lps=2000, max_instances=4) as t:
        with pytest.raises(G.GpqError):
            t.restore(snap)
    with G.PholdSession(max_lps=1000, max_instances=4, bucketed=True) as t:
        with pytest.raises(G.GpqError):
            t.restore(snap)
    with G.PholdSession(max_lps=1000, max_instances=4) as t:
        with pytest.raises(G.GpqError):
            t.restore(snap[:-5])


@pytest.mark.parametrize("shape", [
    # (LPs, events per LP, lookahead, end time) of the runs; capacity; insert capacity; lanes
    ([(700, 44, 30.0, 90.0), (61, 46, 30.0, 90.0), (33, 1, 0.3, 9.0)], 256, 128, 8),  # about a list of safe events
    ([(40, 200, 6.0, 30.0), (9, 130, 0.01, 0.5)], 512, 400, 16),                      # more than a list
    ([(3, 740, 9.0, 30.0), (2, 1000, 9.0, 30.0), (5, 16, 0.5, 20.0)], 2048, 1150, 32),  # about and above the wide list
    ([(20001, 24, 0.4, 4.0), (3, 8, 2.0, 8.0), (500, 20, 0.001, 0.05)], 64, 64, 8),   # eight LPs a turn; idle LPs
    ([(5, 4, 1.0, 10.0 + 0.1 * i) for i in range(300)], 64, 64, 4),                   # more runs than the bounds' table
])
def test_selection_sizes(gpu_lib, shape):
    """Windows whose safe events fit an LP's list, outgrow it and outgrow the warp's space."""
    runs, capacity, insert, lanes = shape
    cfgs = [G.make_phold_config(L, per, la, T, 70 + i) for i, (L, per, la, T) in enumerate(runs)]
    with G.PholdSession(max_lps=sum(c.num_lps for c in cfgs), max_instances=len(cfgs), capacity=capacity,
                        insert_capacity=insert, lanes_per_lp=lanes) as s:
        slot_of = {s.admit(c): i for i, c in enumerate(cfgs)}
        s.step(3)  # then the rest: rings left by one launch, taken up by the next
        s.step(0)
        got = {slot_of[sl]: r for sl, r in s.collect()}
    for i, c in enumerate(cfgs):
        alone = G.make_phold_config(c.num_lps, c.events_per_lp, c.lookahead, c.end_time, c.seed, queue="hq",
                                    capacity=capacity)
        with G.Phold(alone) as h:
            h.populate()
            h.run()
            _same(got[i], h.result())


def test_insert_capacity_too_large_is_refused(gpu_lib):
    with pytest.raises(G.GpqError):
        G.PholdSession(max_lps=8, max_instances=1, insert_capacity=2048, lanes_per_lp=8)
    G.PholdSession(max_lps=8, max_instances=1, insert_capacity=1024, lanes_per_lp=32).close()
