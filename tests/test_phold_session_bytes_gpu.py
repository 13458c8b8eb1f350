"""The memory that a session of PHOLD runs says it takes is what it takes."""
import pytest

import gpupq_b200 as G


@pytest.mark.gpu
@pytest.mark.parametrize("bucketed", [False, True])
def test_bytes_cover_what_a_session_allocates(gpu_lib, bucketed):
    import torch
    lps = 1 << 24
    if bucketed:
        kw, said = dict(buckets=8, bucket_slots=8), gpu_lib.gpq_phold_session_bytes_bucketed(lps, 8, 8, 1)
    else:
        kw, said = dict(capacity=8, insert_capacity=1), gpu_lib.gpq_phold_session_bytes(lps, 8, 1, 1)
    G.PholdSession(max_lps=1, max_instances=1, bucketed=bucketed, **kw).close()  # the module's own memory
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with G.PholdSession(max_lps=lps, max_instances=1, bucketed=bucketed, **kw):
        took = before - torch.cuda.mem_get_info()[0]
    # an allocation of its own is rounded up to 2 MB, and there are about 20; a word per LP is 64 MB
    assert took - (44 << 20) <= said <= took + (44 << 20), (said, took)
