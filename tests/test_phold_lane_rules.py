"""The rules that choose a PHOLD run's lanes per LP: on which side of each of their bounds a
configuration lies, and on the GPU that the run takes the form that the rule names."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import gpupq_b200 as G
from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path_factory.mktemp("rules") / "phold_rules_driver")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "gpupq_b200", "csrc"), "-I",
                           os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                           os.path.join(HERE, "cpp", "phold_rules_driver.cpp"), "-o", exe])

    def ask(cases):
        text = "".join(" ".join(str(x) for x in c) + "\n" for c in cases)
        out = subprocess.run([exe], input=text, capture_output=True, text=True, check=True).stdout.split("\n")
        return [tuple(int(x) for x in line.split()) for line in out[:len(cases)]]

    return ask


def test_local_array_lanes(rules):
    """Lookahead 1: half of an LP's events lie in a window."""
    want = {
        0: {1: (32, 32, 32), 2048: (32, 32, 32), 2049: (16, 16, 32), 3552: (16, 16, 32), 3553: (16, 16, 16),
            4096: (16, 16, 16), 4097: (8, 16, 16), 7104: (8, 16, 16), 7105: (8, 8, 8), 14208: (8, 8, 8),
            14209: (8, 8, 16), 21312: (8, 8, 16), 21313: (8, 8, 8), 65536: (8, 8, 8)},
        1: {1: (32, 32, 32), 2048: (32, 32, 32), 2049: (16, 16, 32), 3552: (16, 16, 32), 3553: (16, 16, 16),
            4096: (16, 16, 16), 4097: (8, 8, 8), 7104: (8, 8, 8), 7105: (8, 8, 8), 14208: (8, 8, 8),
            14209: (8, 8, 8), 21312: (8, 8, 8), 21313: (8, 8, 8), 65536: (8, 8, 8)},
    }
    for mode, rows in want.items():
        for lps, lanes in rows.items():  # just below 2.5 events, from 2.5 on, from 5 on
            got = rules([(mode, lps, 4, 1.0), (mode, lps, 5, 1.0), (mode, lps, 10, 1.0)])
            assert tuple(g[0] for g in got) == lanes, (mode, lps)
            assert rules([(mode, lps, 9, 1.0)])[0][0] == lanes[1]
    for lps in (4097, 7104, 14209, 21312):  # unordered arrays: below 8 events and from 8 on
        assert [g[0] for g in rules([(1, lps, 15, 1.0), (1, lps, 16, 1.0)])] == [8, 16]


def test_splay_lanes(rules):
    for lps, lanes in ((1, 32), (4736, 32), (4737, 16), (9472, 16), (9473, 8), (18944, 8), (18945, 4), (37888, 4),
                       (37889, 1), (1 << 24, 1)):
        assert rules([(0, lps, 8, 1.0)])[0][1] == lanes


def test_heap_form(rules):
    for lps, per, warp in ((1, 1, 1), (1024, 1, 1), (1025, 1, 0), (1025, 2, 1), (4096, 3, 0), (4096, 4, 1), (4097, 4, 0),
                           (4097, 14, 0), (4097, 15, 1), (65536, 14, 0), (65536, 15, 1)):
        assert rules([(0, lps, per, 1.0)])[0][2] == warp, (lps, per)


@pytest.mark.gpu
@pytest.mark.parametrize("queue,mode,lps,per,lanes", [
    ("laq", 0, 2048, 9, 32), ("laq", 0, 2049, 9, 16), ("laq", 0, 4097, 4, 8), ("laq", 0, 4097, 9, 16),
    ("laq", 1, 2048, 9, 32), ("laq", 1, 2049, 9, 16), ("laq", 1, 4097, 15, 8), ("laq", 1, 4097, 16, 16),
    ("lsq", 0, 1024, 5, 32), ("lsq", 0, 4737, 5, 16), ("lsq", 0, 9473, 5, 8),
    ("lhq", 0, 1024, 1, 32), ("lhq", 0, 1025, 1, 8),
])
def test_runs_take_the_form(gpu_lib, queue, mode, lps, per, lanes):
    """A grid below the most that fits has a CTA of 256 threads for 256 / lanes LPs."""
    cfgd = dict(num_lps=lps, events_per_lp=per, lookahead=1.0, end_time=4.0, seed=lps + per, dest_mode=0)
    o = O.phold(O.make_cfg(**cfgd), 8)
    with G.Phold(G.make_phold_config(**cfgd, queue=queue, laq_mode=mode, loop="persistent")) as h:
        h.populate()
        h.run()
        r, s, info = h.result(), h.lp_stats(), h.launch_info()
    assert info["block"] == 256 and info["grid"] == -(-lps // (256 // lanes))
    assert r["status_code"] == 0 and r["committed"] == o["committed"]
    for k in ("count", "csum", "ohash"):
        assert np.array_equal(s[k], o[k]), k
