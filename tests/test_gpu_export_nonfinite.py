"""Exports of a tree built or refitted over non-finite vertices: crt_scene_check reports those, and the export
returns the tree, its leaves' boxes those of the coordinates that are numbers."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 700, 60_000])
@pytest.mark.parametrize("rebuild", [False, True])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e38])
@pytest.mark.parametrize("corners", [1, 3])  # (three: no coordinate of the triangle's box is a number)
def test_export(cuda, n, rebuild, bad, corners):
    import crt
    from crt import data
    m = data.soup(n, seed=n)
    s = crt.Scene(m)
    v = m.verts.copy()
    tri = np.array([n // 2, n - 1])
    v[m.vidx[tri, :corners], 2] = bad
    s.set_vertices(v, rebuild=rebuild)
    e = s.export()
    with pytest.raises(crt.CrtError) as err:
        s.check()
    assert err.value.status == 1
    ids = e["ids"].view(np.uint32).astype(np.int64)
    assert_equal(np.sort(ids), np.arange(n), "ids")
    t = v[m.vidx[ids]]
    leaf = e["node_boxes"].reshape(-1, 6)[n - 1:]
    np.testing.assert_array_equal(leaf[:, :3], np.fmin.reduce(t, 1))
    np.testing.assert_array_equal(leaf[:, 3:], np.fmax.reduce(t, 1))
