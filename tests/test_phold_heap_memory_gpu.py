"""A heap queue of the default node size takes one root for up to 4 M items, and the reference's
256 K nodes where the memory for that root, or for the rest of the handle next to it, is not
there: what fits with such nodes is never refused."""
import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu


def test_default_node_size_with_little_memory(gpu_lib):
    import torch
    cfgd = dict(num_lps=65536, events_per_lp=40, lookahead=0.4, end_time=1.2, seed=3, dest_mode=1, ring_width=7)

    def run(**kw):
        before = torch.cuda.mem_get_info()[0]
        with G.Phold(G.make_phold_config(**cfgd, queue="hq", **kw)) as h:
            took = before - torch.cuda.mem_get_info()[0]
            h.populate()
            h.run()
            r = h.result()
        return {k: r[k] for k in ("committed", "steps", "pending", "pending_csum", "digest", "status_code")}, took

    want, _ = run()
    _, root = run()
    got, nodes = run(node_size=1 << 18)
    assert want["status_code"] == 0 and got == want
    assert root > 2 * nodes
    for leave in (root - (60 << 20), root // 2 + nodes // 2, nodes + (64 << 20)):
        held = []
        try:
            while torch.cuda.mem_get_info()[0] > leave + (4 << 20):
                free = torch.cuda.mem_get_info()[0]
                held.append(torch.empty(max(min(free - leave, 16 << 30), 2 << 20), dtype=torch.uint8, device="cuda"))
            got, took = run()
            assert got == want and took < 2 * nodes
        finally:
            held.clear()
            torch.cuda.empty_cache()
