"""The quantised wide nodes at the edges of their range: coordinates near the float limits, flat and far-off
meshes, and triangle counts around one refit block.  The export refuses a tree with a slot that does not
contain its node's exact box, and the traces must equal the oracle's bit for bit."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


def _mesh(kind, n, rng):
    from crt import data
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    v = c + rng.normal(0.0, 0.05, (n, 3, 3))
    if kind == "flat":  # one plane: a zero extent on an axis of every node
        v[..., 2] = -3.0
    elif kind == "far":  # boxes of a few hundred ulps
        v = v * 1e-2 + np.array([1000.0, -2000.0, 3000.0])
    elif kind == "zero":  # every coordinate 0 on two axes
        v[..., 1:] = 0.0
    elif kind != "unit":
        v = v * float(kind)
    v = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1))
    return data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])


@pytest.mark.parametrize("n", [2, 3, 511, 512, 513, 1500])
@pytest.mark.parametrize("kind", ["unit", "flat", "far", "zero", "1e-30", "1e-18", "1e16", "1e33", "4e36"])
def test_quantised_nodes(cuda, kind, n):
    import crt
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(n)
    m = _mesh(kind, n, rng)
    g, o = crt.Scene(m), OracleScene(m)
    ge, oe = g.export(), o.export()  # (the export checks every slot against the exact boxes)
    for k in ("codes", "ids", "nodes", "node_boxes"):
        assert_equal(ge[k], oe[k], k)
    lo, hi = m.verts.astype(np.float64).min(0), m.verts.astype(np.float64).max(0)
    org = rng.uniform(lo - 0.1 * (hi - lo), hi + 0.1 * (hi - lo), (600, 3))
    to = m.verts[m.vidx[rng.integers(0, n, 600)]].astype(np.float64).mean(1)
    d = to - org
    d[:100] = rng.normal(size=(100, 3))
    ln = np.abs(d).max(1, keepdims=True)
    d = d / np.where(ln > 0, ln, 1.0)
    d[100:110] = np.eye(3)[np.arange(10) % 3]
    d /= np.linalg.norm(d, axis=1, keepdims=True) + (np.abs(d).max(1, keepdims=True) == 0)
    rays = np.hstack([org, d])
    for any_hit in (False, True):
        gi, gt = g.trace(rays, any_hit=any_hit)
        oi, ot, _ = o.trace(rays, any_hit=any_hit)
        assert_equal(gi, oi, f"ids any={any_hit}")
        assert_equal(gt, ot, f"t any={any_hit}")
    g.check()
    # a refit writes the same nodes again
    g.refit()
    assert_equal(g.export()["node_boxes"], oe["node_boxes"], "refit boxes")
