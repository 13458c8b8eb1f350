"""Reference-semantics A* on the GPU against its CPU oracle, every agent bit for bit
(found, the goal's half-precision f, pops, rounds), with any number of concurrent slots:
agents are independent, so the slot schedule changes nothing."""
import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(m, agents, slots, open_capacity=0):
    with G.AStarRef(m.shape[1], m.shape[0], slots=slots, open_capacity=open_capacity) as a:
        got = a.solve(m, agents)
    _, want = O.astar_ref(m, agents, threads=8)
    assert (got["status"] == 0).all()
    for k in ("found", "pops", "rounds"):
        assert np.array_equal(got[k], want[k]), k
    assert np.array_equal(got["cost"].view(np.uint32), want["cost"].view(np.uint32))
    return got


@pytest.mark.parametrize("w,h,frac,slots", [(64, 64, 0.2, 64), (128, 96, 0.25, 7), (256, 256, 0.2, 2048),
                                            (256, 256, 0.2, 1), (37, 211, 0.1, 300)])
def test_agents_match_oracle(gpu_lib, w, h, frac, slots):
    m = G.astar_ref_map(w, h, frac, 1.0, seed=w + h)
    n = 64 if slots == 1 else 600
    agents = G.astar_ref_agents(m, n, seed=7)
    r = _check(m, agents, slots)
    assert r["found"].sum() > n // 2


def test_edge_agents(gpu_lib):
    m = np.zeros((16, 16), np.uint8)
    m[:, 8] = 1
    agents = np.array([(5 * 16 + 2, 5 * 16 + 2), (0, 255), (0, 15 * 16 + 7)], G.ASTAR_REF_AGENT_DTYPE)
    r = _check(m, agents, slots=2)
    assert list(r["found"]) == [1, 0, 1]


def test_open_list_overflow_is_reported(gpu_lib):
    m = np.zeros((64, 64), np.uint8)
    agents = np.array([(0, 64 * 64 - 1)], G.ASTAR_REF_AGENT_DTYPE)
    with G.AStarRef(64, 64, slots=1, open_capacity=16) as a:
        r = a.solve(m, agents)
    assert r[0]["status"] == 3  # GPQ_ERR_QUEUE_FULL


@pytest.mark.parametrize("w,h,frac", [(1, 300, 0.0), (300, 1, 0.0), (9, 8, 0.1), (200, 200, 0.0), (2048, 2048, 0.2),
                                      (8192, 512, 0.2), (8193, 9, 0.1), (2049, 2048, 0.2)])
def test_vertex_forms(gpu_lib, w, h, frac):
    """Sizes at the edges of the packed vertex word (up to 22 coordinate bits, sides up to
    8,192; beyond them the general form) and open lists of one to thousands of vertices:
    agents between nearby cells all over the map, one that starts on its goal, and -- on the
    small maps -- one whose goal is walled in, so that the whole map is searched."""
    m = G.astar_ref_map(w, h, frac, 1.0, seed=w + h) if frac else np.zeros((h, w), np.uint8)
    rng = np.random.default_rng(w * 7 + h)
    free = lambda x, y: m[y, x] == 0  # noqa: E731
    pairs = []
    while len(pairs) < 40:
        x0, y0 = int(rng.integers(w)), int(rng.integers(h))
        x1, y1 = (int(np.clip(v + rng.integers(-40, 41), 0, n - 1)) for v, n in ((x0, w), (y0, h)))
        if free(x0, y0) and free(x1, y1):
            pairs.append((y0 * w + x0, y1 * w + x1))
    pairs.append((pairs[0][0], pairs[0][0]))
    if w == 200:
        gx, gy = 150, 40
        m[gy - 1:gy + 2, gx - 1:gx + 2] = 1
        m[gy, gx] = 0
        pairs.append((120 * w + 17, gy * w + gx))
    _check(m, np.array(pairs, G.ASTAR_REF_AGENT_DTYPE), slots=7)
