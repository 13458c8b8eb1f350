"""Launch shapes of the grid search: the CTAs per SM that the frontier-list form holds, and a
shape read back from one search and asked for in the next."""
import numpy as np
import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile,block", [(16, 256), (8, 256), (64, 128)])
def test_four_list_ctas_an_sm(gpu_lib, tile, block):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    grids = G.astar_queries(3, 40, 8, 64, 300, 0.1, 0.3)
    with G.AStar(tile=tile, block_threads=block, ctas_per_sm=4, frontier_capacity=1024) as a:
        a.solve(grids)
        assert a.stats()["grid"] == 4 * sms


@pytest.mark.parametrize("cfg", [dict(), dict(tile=64), dict(tile=32), dict(tile=16), dict(tile=32, tile_worker=1)])
def test_the_block_read_back_may_be_asked_for(gpu_lib, cfg):
    grids = G.astar_queries(3, 40, 8, 64, 300, 0.1, 0.3)
    with G.AStar(**cfg) as a:
        want = a.solve(grids)
        block = a.stats()["block"]
    with G.AStar(**cfg, block_threads=block) as a:
        got = a.solve(grids)
        assert a.stats()["block"] == block
    for k in ("cost", "expanded", "gsum", "path_len", "path_hash", "status"):
        assert np.array_equal(got[k], want[k])
    cells = 1 << 20
    G.AStarSession(cells, 4096, 4, **cfg, block_threads=block).close()


@pytest.mark.parametrize("cfg", [dict(tile=64, tile_worker=1), dict(tile=32), dict(tile=16), dict(tile=128)])
def test_512_threads_are_for_swept_tiles_of_64(gpu_lib, cfg):
    with pytest.raises(G.GpqError):
        G.AStar(**cfg, block_threads=512)
