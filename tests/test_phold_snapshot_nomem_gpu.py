"""A restore that is refused for want of device memory leaves the handle, and the library's
other calls on the thread, as they were."""
import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu


def test_restore_without_memory_for_the_other_layout(gpu_lib):
    import torch
    cfgd = dict(num_lps=65536, events_per_lp=40, lookahead=0.4, end_time=2.0, seed=3, dest_mode=1, ring_width=7)

    def run(h):
        h.run()
        r = h.result()
        return {k: r[k] for k in ("committed", "steps", "pending", "pending_csum", "digest", "status_code")}

    def snap(node_size):
        with G.Phold(G.make_phold_config(**cfgd, queue="hq", node_size=node_size)) as h:
            h.populate()
            h.step(2)
            return h.snapshot()

    nodes, root = snap(1 << 18), snap(0)
    at = 8 + G.PholdConfig.node_size.offset
    nodes[at:at + 4] = 0  # as a handle of the default size writes it
    with G.Phold(G.make_phold_config(**cfgd, queue="hq")) as h:
        h.restore(nodes)
        want = run(h)
        assert want["status_code"] == 0
        held = []
        try:
            while True:  # all but 0.4 GB, of which the other layout needs about 0.9
                free = torch.cuda.mem_get_info()[0]
                if free < (400 << 20) + (64 << 20):
                    break
                held.append(torch.empty(min(free - (400 << 20), 16 << 30), dtype=torch.uint8, device="cuda"))
            with pytest.raises(G.GpqError):
                h.restore(root)
            h.populate()
            assert run(h) == want
            h.restore(nodes)
            assert run(h) == want
        finally:
            held.clear()
            torch.cuda.empty_cache()
        h.restore(root)
        assert run(h) == want
