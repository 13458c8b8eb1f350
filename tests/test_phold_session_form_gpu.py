"""The form of a session's rings in its snapshot."""
import struct

import numpy as np
import pytest

import gpupq_b200 as G

FORM_AT = 8 + 4 * 11  # the last word of the snapshot's header


def _form(snap):
    return struct.unpack_from("<I", snap.tobytes(), FORM_AT)[0]


@pytest.mark.gpu
def test_snapshot_names_the_form_of_its_rings(gpu_lib):
    """Rings in any order are not what a reader of sorted rings takes (form 1); such a reader's
    own snapshots, whose rings are sorted, are still restored.  Time buckets are as before."""
    runs = [G.make_phold_config(300 + 50 * i, 16, 0.5, 12.0, 5 + i) for i in range(3)]

    def finish(s, slots):
        s.step(0)
        got = dict(s.collect())
        return [(got[i].committed, got[i].steps, got[i].pending, got[i].digest, got[i].status) for i in slots]

    for bucketed, form in ((False, 2), (True, 1)):
        kw = dict(max_lps=2000, max_instances=4, bucketed=bucketed)
        with G.PholdSession(**kw) as s:
            slots = [s.admit(c) for c in runs]
            s.step(0 if bucketed else 1)
            fresh = s.snapshot()
            s.step(4)
            later = s.snapshot()
            want = finish(s, slots) if not bucketed else None
        assert _form(fresh) == _form(later) == form
        if bucketed:
            continue
        for snap in (fresh, later):
            old = snap.copy()
            old[FORM_AT:FORM_AT + 4] = np.frombuffer(struct.pack("<I", 1), np.uint8)
            other = snap.copy()
            other[FORM_AT:FORM_AT + 4] = np.frombuffer(struct.pack("<I", 3), np.uint8)
            with G.PholdSession(**kw) as t:
                with pytest.raises(G.GpqError):
                    t.restore(other)
                for b in (snap, old):
                    t.restore(b)
                    assert finish(t, slots) == want
