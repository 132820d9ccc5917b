"""Zeros of both signs in an exported tree.  The device's min and max order -0 below +0 whatever their operands' order,
so the host's unions of the leaves' boxes have to as well: the export must neither refuse such a tree nor return
other zeros than the device's boxes hold."""
import ctypes
import itertools

import numpy as np
import pytest

from conftest import assert_equal

EXPORT_TREE = "_ZN3crt11export_treeEiPKjPKNS_5WNodeEPKNS_7LeafTriEPKfPiPf"
EMPTY = -(1 << 31)
WNODE = np.dtype([("o", "<f4", 3), ("s15", "<f4", 3), ("lo", "<u4", 3), ("hi", "<u4", 3), ("code", "<i4", 4)])


def _export_two(z):
    """A tree of two triangles with corner depths z[0..5] (all zeros), as the device holds it, through the host's
    export: its boxes, or None when it is refused."""
    import crt
    leaves = np.zeros((2, 3, 4), np.float32)
    leaves[0, :, :2] = [(0, 0), (0.5, 0), (0, 0.5)]
    leaves[1, :, :2] = [(0.5, 0.5), (1, 0.5), (0.5, 1)]
    leaves[:, :, 2] = np.asarray(z, np.float32).reshape(2, 3)
    node = np.zeros(1, WNODE)
    # quanta of 2^-7 in x and y, of 2^-63 in z; s15 is 2^15 quanta and o + s15 the least plane
    node["s15"] = [2.0 ** 8, 2.0 ** 8, 2.0 ** -48]
    node["o"] = -node["s15"]
    for slot, (lo, hi) in {0: (0, 64), 2: (64, 128)}.items():
        for k in range(2):
            node["lo"][0, k] |= lo << (8 * slot)
            node["hi"][0, k] |= hi << (8 * slot)
    node["lo"][0] |= 0xFF00FF00  # empty slots: 255 and 0
    node["code"] = [~0, EMPTY, ~1, EMPTY]
    parent = np.array([0, 1 << 31, 0], np.uint32)  # the root; leaf 0 is its left child, leaf 1 its right one
    neg = np.signbit(z)
    root = np.array([0, 0, -0.0 if neg.any() else 0.0, 1, 1, -0.0 if neg.all() else 0.0], np.float32)
    nodes, boxes = np.zeros(9, np.int32), np.zeros((3, 6), np.float32)
    fn = getattr(crt.lib(), EXPORT_TREE)
    fn.restype = ctypes.c_bool
    ptr = [ctypes.c_void_p(a.ctypes.data) for a in (parent, node, leaves, root, nodes, boxes)]
    return boxes if fn(ctypes.c_int(2), *ptr) else None


@pytest.mark.parametrize("z", list(itertools.product([0.0, -0.0], repeat=6)))
def test_zeros_keep_the_device_order(built, z):
    boxes = _export_two(z)
    assert boxes is not None, "refused"
    neg = np.signbit(z)
    want = [(neg.any(), neg.all()), (neg[:3].any(), neg[:3].all()), (neg[3:].any(), neg[3:].all())]
    assert_equal(np.signbit(boxes[:, [2, 5]]), np.array(want), "signs of the zero planes")


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 40, 1500])
def test_flat_mesh_at_both_zeros(cuda, n):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(n)
    v = rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.normal(0.0, 0.05, (n, 3, 3))
    v[..., 2] = np.where(rng.random((n, 3)) < 0.5, 0.0, -0.0)
    v = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    m = data.Mesh(v, idx, np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1)), idx.copy(),
                  np.zeros(n, np.int32), data.lambert_material()[None])
    want = OracleScene(m).export()["node_boxes"]
    view = (data.Camera(fov=60.0), data.Light(), 16, 16, 1)
    batch = crt.Batch([m], [view])
    batch.run(np.zeros((256, 3), np.uint8))
    for e in (crt.Scene(m).export(), batch.export(0)):
        assert_equal(e["node_boxes"], want, "boxes")
        z = v[e["ids"].view(np.uint32).astype(np.int64)[:, None] * 3 + np.arange(3), 2]
        leaf = np.signbit(e["node_boxes"].reshape(-1, 6)[n - 1:, [2, 5]])
        assert_equal(leaf, np.stack([np.signbit(z).any(1), np.signbit(z).all(1)], 1), "signs of the leaves' zeros")
