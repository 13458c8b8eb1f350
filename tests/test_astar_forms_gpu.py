"""Launch shapes of the grid search: the CTAs per SM that the frontier-list form holds."""
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
