"""A refused dequeue leaves a queue object as it was, and its work is finished when it
returns: a retry on another stream gets every item."""
import ctypes
import math

import numpy as np
import pytest

import gpupq_b200 as G

pytestmark = pytest.mark.gpu


def _dequeue(q, bound, most, out, cap, stream):
    n = ctypes.c_uint64()
    st = G.lib().gpq_queue_dequeue(q._h, bound, most, ctypes.c_void_p(out.ctypes.data), cap, ctypes.byref(n),
                                   ctypes.c_void_p(stream.cuda_stream))
    return st, n.value


@pytest.mark.parametrize("kind", ["laq", "gaq"])
@pytest.mark.parametrize("lps,n", [(700, 5000), (8192 * 32, 40)])
def test_refused_then_retried_on_another_stream(gpu_lib, kind, lps, n):
    import torch
    rng = np.random.default_rng(n)
    have = np.zeros(n, G.ITEM_DTYPE)
    have["ts"] = rng.standard_exponential(n, dtype=np.float32)
    have["lp"] = rng.integers(0, lps, n)
    have["id"] = rng.permutation(n)
    want = have[np.lexsort((have["id"], have["ts"].view(np.uint32), have["lp"]))]
    first = np.append(True, want["lp"][1:] != want["lp"][:-1])
    # work of others fills the GPU and the retry's stream goes first: what the refused call
    # leaves unfinished on its own stream comes after the retry
    streams = [torch.cuda.Stream(), torch.cuda.Stream(priority=-1)]
    load, a = torch.cuda.Stream(), torch.ones(4096, 4096, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    out = np.zeros(n, G.ITEM_DTYPE)
    with G.Queue(kind, lps, capacity=32, insert_capacity=32) as q:
        for turn in range(10):
            q.insert(have)
            q.post()
            with torch.cuda.stream(load):
                for _ in range(10):
                    torch.matmul(a, a)
            st, total = _dequeue(q, math.inf, 0, out, n - 1, streams[0])
            assert st != 0 and total == n
            parts = []
            for most in (1, 0) if turn % 2 else (0,):
                st, total = _dequeue(q, math.inf, most, out, n, streams[1])
                assert st == 0
                parts.append(out[:total].copy())
            assert sum(len(p) for p in parts) == n
            if turn % 2:
                assert np.array_equal(parts[0], want[first])
                assert np.array_equal(parts[1], want[~first])
            else:
                assert np.array_equal(parts[0], want)
            assert q.get_min() == math.inf
