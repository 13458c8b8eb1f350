"""Queue objects at the sizes where their dequeue and insert change form: LPs around a
CTA's share, items around the page-locked buffer's, limits around a lane group's width,
outputs that are too small; against numpy's sort by (LP, timestamp, id)."""
import math

import numpy as np
import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu


def _items(rng, lps, n, base=0.0, first=0):
    a = np.zeros(n, G.ITEM_DTYPE)
    a["ts"] = np.float32(base) + np.round(rng.standard_exponential(n) * 64).astype(np.float32) / np.float32(64)  # ties
    a["lp"] = rng.permutation(np.arange(n, dtype=np.uint32) % np.uint32(lps))
    a["id"] = first + rng.permutation(n)
    a["aux"] = rng.integers(0, 1 << 30, n)
    return a


def _order(a):
    return a[np.lexsort((a["id"], a["ts"].view(np.uint32), a["lp"]))]


def _take(have, bound, most):
    """What a dequeue returns, and what stays."""
    s = _order(have)
    first = np.searchsorted(s["lp"], s["lp"], side="left")
    ok = s["ts"] < np.float32(bound)
    if most:
        ok &= (np.arange(len(s)) - first) < most
    return s[ok], s[~ok]


@pytest.mark.parametrize("kind", ["laq", "gaq"])
@pytest.mark.parametrize("lps,n", [(1, 1), (1, 40), (31, 300), (32, 320), (33, 330), (700, 8191), (700, 8192), (700, 8193),
                                   (8192, 20000), (8193, 20000), (20011, 60000)])
@pytest.mark.parametrize("most", [0, 1, 8, 9])
def test_dequeue_sizes(gpu_lib, kind, lps, n, most):
    rng = np.random.default_rng(lps + n)
    have = _items(rng, lps, n)
    with G.Queue(kind, lps, capacity=128, insert_capacity=64) as q:
        q.insert(have)
        q.post_init()
        for w in range(3):
            assert q.get_min() == (float(have["ts"].min()) if len(have) else math.inf)
            bound = float(np.float32(0.3 + 0.4 * w))
            want, have = _take(have, bound, most)
            if len(want) > 1:
                with pytest.raises(G.GpqError):
                    q.dequeue(bound, most, capacity=len(want) - 1)
            got = q.dequeue(bound, most, capacity=max(1, len(want)))
            assert np.array_equal(got, want)
            more = _items(rng, lps, n // 4, 0.2 * w, n * (w + 1))
            if len(more):
                q.insert(more)
            q.post()
            have = np.concatenate([have, more])
        got = q.dequeue(math.inf)
        assert np.array_equal(got, _take(have, math.inf, 0)[0])
        assert len(q.dequeue(math.inf)) == 0 and q.get_min() == math.inf
        assert q.counts() == (n + 3 * (n // 4), n + 3 * (n // 4))


def test_more_lps_than_counted(gpu_lib):
    lps = 8192 * 32 + 1
    rng = np.random.default_rng(3)
    have = _items(rng, lps, 30000)
    have["lp"][:2] = (0, lps - 1)
    with G.Queue("laq", lps, capacity=64, insert_capacity=64) as q:
        q.insert(have)
        q.post()
        want, have = _take(have, 0.5, 0)
        assert np.array_equal(q.dequeue(0.5), want)
        assert np.array_equal(q.dequeue(math.inf), _order(have))


@pytest.mark.parametrize("kind", ["laq", "lhq"])
def test_insert_error_is_reported_once(gpu_lib, kind):
    a = np.zeros(40, G.ITEM_DTYPE)
    a["id"] = np.arange(40)
    with G.Queue(kind, 2, capacity=64, insert_capacity=32) as q:
        q.insert(a)
        with pytest.raises(G.GpqError):
            q.post()
        q.post()
        assert len(q.dequeue(math.inf)) == 32
