"""A* tile visits in each of their forms -- sweeps by CTAs of several sizes, frontier lists --
at grid sides around the tile's, both connectivities, narrow and wide windows and densities
up to where paths wind, against the oracle."""
import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FIELDS = ("cost", "expanded", "gsum", "path_len", "path_hash")


def _check(res, grids):
    for i, g in enumerate(grids):
        want = O.astar({k: int(g[k]) for k in O.ASTAR_FIELDS})
        assert res[i]["status"] == 0, (i, int(res[i]["status"]))
        for k in FIELDS:
            assert int(res[i][k]) == want[k], (i, k, int(res[i][k]), want[k])


def _grids():
    out = []
    for conn in (4, 8):
        for w, h in ((1, 1), (1, 200), (200, 1), (31, 33), (32, 32), (33, 15), (63, 65), (64, 64), (65, 64), (130, 17),
                     (97, 129)):
            out.append(G.astar_grid(w, h, 0.15, 5 * w + h, conn=conn))
            out.append(G.astar_grid(w, h, 0.0, 1, conn=conn, start=w * h - 1, goal=0))
        for dens in (0.1, 0.3, 0.38, 0.45):  # beyond about 0.4 most goals are walled off
            out += [G.astar_queries(77, 1, conn, 150, 300, dens, dens, first=i) for i in range(3)]
    return np.concatenate(out)


@pytest.mark.parametrize("tile,block,worker", [(64, 0, 0), (64, 256, 0), (64, 128, 0), (32, 0, 0), (32, 128, 0),
                                               (32, 64, 0), (16, 64, 0), (32, 64, 1)])
@pytest.mark.parametrize("window", [1, 7, 300])
def test_tile_visit_forms(gpu_lib, tile, block, worker, window):
    grids = _grids()
    with G.AStar(tile=tile, block_threads=block, tile_worker=worker, window=window) as a:
        for _ in range(2):
            _check(a.solve(grids), grids)


def test_items_above_the_frontier_capacity(gpu_lib):
    grids = _grids()
    with G.AStar(tile=64, window=1000, frontier_capacity=64, inbox_capacity=1 << 13) as a:
        _check(a.solve(grids), grids)
