"""Which decode passes of a Llama-format model are captured and replayed (csrc/graph_slots.h), walked on the host through
cpmcu_debug_decode_graphs.  No GPU."""
import ctypes
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cpm.cu_b200"))
PLAIN, CAPTURE, REPLAY = 0, 1, 2


def acts(shapes):
    import __graft_entry__ as entry
    import cpmcu.C as C
    if not os.path.exists(C.lib_path()):
        entry.build()
    s, out = np.asarray(shapes, dtype=np.int32), np.full(len(shapes), -1, dtype=np.int32)
    C.call("cpmcu_debug_decode_graphs", ctypes.c_void_p(s.ctypes.data), len(s), ctypes.c_void_p(out.ctypes.data))
    return out


def test_a_shape_is_captured_the_second_time():
    assert acts([2, 3, 2, 2, 3, 2, 3]).tolist() == [PLAIN, PLAIN, CAPTURE, REPLAY, CAPTURE, REPLAY, REPLAY]


def test_more_shapes_than_slots_in_turn_cost_no_captures():
    """Trees of 40 sizes one after the other, fifty times: the first 16 keep their graphs, the others run launch by launch."""
    a = acts(list(range(40)) * 50).reshape(50, 40)
    assert (a[0] == PLAIN).all() and (a[1, :16] == CAPTURE).all() and (a == CAPTURE).sum() == 16
    assert (a[2:, :16] == REPLAY).all() and (a[:, 16:] == PLAIN).all()


def test_random_shapes_cost_few_captures():
    shapes = np.random.default_rng(0).integers(0, 128, 4000)
    a = acts(shapes)
    assert (a == CAPTURE).sum() <= 16 + 16 * 4000 // 256


def test_a_graph_that_is_left_alone_gives_its_slot_up():
    a = acts(list(range(16)) * 2 + [100] * 400 + list(range(15, -1, -1)))
    new = a[32:432]
    at = int(np.argmax(new == CAPTURE))
    assert (new[:at] == PLAIN).all() and at <= 256 and (new[at + 1:] == REPLAY).all()
    # one slot went, the one that had been replayed longest ago
    assert a[432:].tolist() == [REPLAY] * 15 + [PLAIN]


def test_every_replay_follows_a_capture_of_its_shape():
    shapes = np.random.default_rng(1).zipf(1.3, 5000) % 128
    held = set()
    for s, a in zip(shapes.tolist(), acts(shapes).tolist()):
        if a == REPLAY:
            assert s in held
        if a == CAPTURE:
            assert s not in held or len(held) > 16   # evicted in between
            held.add(s)
