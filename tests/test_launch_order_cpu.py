"""What LaunchOrder (csrc/launch_order.h) says has ended when a launch starts, through cpmcu_debug_launch_order, against launches that take any
time: a launch starts once every CTA of its predecessor has let it, at the predecessor's start or, where it holds its successor back, when its
wait for its own predecessor is over.  No GPU."""
import ctypes
import itertools
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cpm.cu_b200"))


def ended(holds):
    import __graft_entry__ as entry
    import cpmcu.C as C
    if not os.path.exists(C.lib_path()):
        entry.build()
    h, out = np.asarray(holds, dtype=np.int32), np.full(len(holds), -1, dtype=np.int32)
    C.call("cpmcu_debug_launch_order", ctypes.c_void_p(h.ctypes.data), len(h), ctypes.c_void_p(out.ctypes.data))
    return out.tolist()


def schedule(holds, lasting):
    """Start and end of every launch; all of them wait for their predecessor before their last work."""
    start, end = [0.0], [lasting[0]]
    for i in range(1, len(holds)):
        before = end[i - 2] if i > 1 else 0.0
        start.append(max(start[i - 1], before) if holds[i - 1] else start[i - 1])
        end.append(max(start[i], end[i - 1]) + lasting[i])
    return start, end


@pytest.mark.parametrize("n", [1, 2, 3, 7])
def test_every_order(n):
    g = np.random.default_rng(n)
    for holds in itertools.product((0, 1), repeat=n):
        got, surely = ended(holds), list(range(n))
        for _ in range(40):
            start, end = schedule(holds, g.exponential(1.0, n) + 0.01)
            surely = [min(s, sum(e <= start[i] for e in end[:i])) for i, s in enumerate(surely)]
        assert got == surely, holds


def test_chains_of_a_token():
    # norm, router (holds), gate/up (holds), down, sum: gate/up has the norm behind it, the down product and the sum the router
    assert ended([0, 1, 1, 0, 0]) == [0, 0, 1, 2, 2]
    # a launch between router and gate/up, or a router that starts its successor at once: nothing has ended
    assert ended([0, 1, 0, 1, 0])[2:4] == [1, 1] and ended([0, 0, 1])[2] == 0
    # queries/keys/values, recurrence's product (holds), norms, splits, step (holds), merge
    assert ended([0, 1, 0, 0, 1, 0]) == [0, 0, 1, 1, 1, 4]
