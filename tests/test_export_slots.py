"""The export's check of the wide nodes: slots that miss a part of their box or that are looser than the packing makes
them are an inconsistent tree (loose ones change no image, they only make every walk longer)."""
import ctypes

import numpy as np
import pytest

EXPORT_TREE = "_ZN3crt11export_treeEiPKjPKNS_5WNodeEPKNS_7LeafTriEPKfPiPf"
EMPTY = -(1 << 31)
WNODE = np.dtype([("o", "<f4", 3), ("s15", "<f4", 3), ("lo", "<u4", 3), ("hi", "<u4", 3), ("code", "<i4", 4)])
PLANES = {0: (0, 64), 2: (64, 128)}  # of two triangles on [0, 0.5] and [0.5, 1], in quanta of 2^-7


def _accepts(planes=PLANES, scale=1.0, code=(~0, EMPTY, ~1, EMPTY), shift=0.0):
    import crt
    leaves = np.zeros((2, 3, 4), np.float32)
    leaves[0, :, :3] = [(0, 0, 0), (0.5, 0, 0.5), (0, 0.5, 0)]
    leaves[1, :, :3] = [(0.5, 0.5, 1), (1, 0.5, 0.5), (0.5, 1, 1)]
    node = np.zeros(1, WNODE)
    node["s15"] = scale * 2.0 ** 8  # 2^15 quanta; o + s15 is the least plane
    node["o"] = shift - node["s15"]
    for slot, (lo, hi) in planes.items():
        node["lo"] |= np.uint32(lo << (8 * slot))
        node["hi"] |= np.uint32(hi << (8 * slot))
    node["lo"] |= np.uint32(0xFF00FF00)
    node["code"] = code
    parent = np.array([0, 1 << 31, 0], np.uint32)
    root = np.array([0, 0, 0, 1, 1, 1], np.float32)
    nodes, boxes = np.zeros(9, np.int32), np.zeros((3, 6), np.float32)
    fn = getattr(crt.lib(), EXPORT_TREE)
    fn.restype = ctypes.c_bool
    return fn(ctypes.c_int(2), *[ctypes.c_void_p(a.ctypes.data) for a in (parent, node, leaves, root, nodes, boxes)])


@pytest.mark.parametrize("what,kw,ok", [
    ("tight", {}, True),
    ("four quanta loose", dict(planes={0: (0, 68), 2: (60, 132)}), True),
    ("five quanta loose above", dict(planes={0: (0, 69), 2: (64, 128)}), False),
    ("five quanta loose below", dict(planes={0: (0, 64), 2: (59, 128)}), False),
    ("all of the node", dict(planes={0: (0, 255), 2: (0, 255)}), False),
    ("misses a part above", dict(planes={0: (0, 63), 2: (64, 128)}), False),
    ("misses a part below", dict(planes={0: (0, 64), 2: (65, 128)}), False),
    ("finer quanta", dict(planes={0: (0, 128), 2: (128, 255)}, scale=0.5), False),  # (255 quanta do not reach 1)
    ("coarser quanta", dict(planes={0: (0, 32), 2: (32, 64)}, scale=2.0), False),
    ("origin above the box", dict(shift=2.0 ** -7), False),
    ("another node's code", dict(code=(~1, EMPTY, ~0, EMPTY)), False),
    ("a filled empty slot", dict(code=(~0, ~0, ~1, EMPTY)), False)])
def test_slots(built, what, kw, ok):
    assert _accepts(**kw) == ok
