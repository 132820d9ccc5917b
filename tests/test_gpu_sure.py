"""The pixel kernels' hits that FP32 settles (certain closest hits, a shadow ray's own triangle) at the edges where it
cannot: coincident and nearly coincident triangles, sheets closer than the FP32 bound, very small and very large
triangles, lights that graze the surface.  Hit ids, t, shadow bits and the image must equal the oracle's."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


def _grid(n, z, jitter, rng):
    """An n x n sheet of quads (two triangles each) facing the camera."""
    t = np.linspace(-1.0, 1.0, n + 1)
    x, y = np.meshgrid(t, t, indexing="ij")
    p = np.stack([x, y, np.full_like(x, z)], -1) + rng.normal(0.0, jitter, x.shape + (3,))
    a, b, c, d = p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]
    return np.concatenate([np.stack([a, b, c], 2).reshape(-1, 3, 3), np.stack([a, c, d], 2).reshape(-1, 3, 3)])


def _scene(kind):
    rng = np.random.default_rng(11)
    if kind == "duplicates":
        return np.repeat(_grid(12, -3.0, 0.05, rng), 3, 0)
    if kind == "sheets":  # closer together than FP32 can tell
        return np.concatenate([_grid(12, -3.0 - 1e-7 * k, 0.0, rng) for k in range(4)])
    if kind == "crossing":  # two sheets that cut each other at a shallow angle
        a, b = _grid(15, -3.0, 0.0, rng), _grid(15, -3.0, 0.0, rng)
        a[..., 2] += 1e-4 * a[..., 0]
        b[..., 2] -= 1e-4 * b[..., 0]
        return np.concatenate([a, b])
    if kind == "fine":
        return _grid(160, -3.0, 1e-4, rng)
    if kind == "coarse":
        return _grid(1, -3.0, 0.0, rng) * np.array([40.0, 40.0, 1.0])
    return _grid(12, -3.0, 0.02, rng) * 1e3  # large coordinates


@pytest.mark.parametrize("kind", ["duplicates", "sheets", "crossing", "fine", "coarse", "large"])
@pytest.mark.parametrize("light", [(2.5, 2.5, -0.5), (5.0, 0.5, -2.5), (5.0, 0.5, -2.4999999), (0.5, 0.5, -9.5)])
@pytest.mark.parametrize("fstop", [np.inf, 2.0])
def test_sure_hits(cuda, kind, light, fstop):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    v = _scene(kind).reshape(-1, 3).astype(np.float32)
    n = len(v) // 3
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1))
    m = data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])
    cam = data.Camera(fov=50.0, focal_point=3.0, fstop=fstop)
    lt = data.Light(position=light)
    w, h, spp = 72, 52, 4
    g, o = crt.Scene(m), OracleScene(m)
    got = g.render(cam, lt, w, h, spp, aux=True, rays=True)
    ref = o.render(cam, lt, w, h, spp=spp, aux=True, rays_in=got["rays"])
    for k in ("hit_id", "hit_t", "shadow"):
        assert_equal(got[k], ref[k], k)
    assert_equal(got["rgb8"], ref["rgb"], "image")
    b = crt.Batch([m], [(cam, lt, w, h, spp)])
    assert_equal(b.run(np.zeros((w * h, 3), np.uint8)), got["rgb8"], "batched image")
    g.check()


@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e3])
@pytest.mark.parametrize("offset", [0.0, 30.0, 3e4])
def test_rays_at_edges(cuda, scale, offset):
    """Rays aimed at edges and corners, on them and beside them by 1e-9 to 1e-4 of a triangle: the FP32 filters'
    error bounds decide which of these take the exact test; closest and any hits must be the oracle's."""
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(3)
    tri = _grid(14, 0.0, 0.02, rng)
    v = (tri.reshape(-1, 3) * scale + offset).astype(np.float32)
    n = len(v) // 3
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1))
    m = data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])
    g, o = crt.Scene(m), OracleScene(m)
    k = 12_000
    t = v.reshape(-1, 3, 3).astype(np.float64)[rng.integers(0, n, k)]
    s = np.where(rng.random(k) < 0.2, 0.0, rng.random(k))[:, None]  # corners, points of edges
    p = t[:, 0] + s * (t[:, 1] - t[:, 0])
    size = np.linalg.norm(t[:, 1] - t[:, 0], axis=1, keepdims=True)
    p = p + rng.normal(size=(k, 3)) * size * 10.0 ** rng.uniform(-9, -4, (k, 1)) * (rng.random((k, 1)) < 0.8)
    d = rng.normal(size=(k, 3))
    d[: k // 4, 2] *= 1e-3  # grazing
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.hstack([p - d * scale * rng.uniform(0.0, 4.0, (k, 1)), d])
    for any_hit in (False, True):
        gi, gt = g.trace(rays, any_hit=any_hit)
        oi, ot, _ = o.trace(rays, any_hit=any_hit)
        assert_equal(gi, oi, f"ids any={any_hit}")
        assert_equal(gt, ot, f"t any={any_hit}")
    g.check()


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("offset", [0.0, 0.3, -700.0])
def test_flat_boxes(cuda, axis, offset):
    """Axis-aligned triangles, whose boxes are flat: rays inside, on and beside their edges, along the axis, across
    it and within the plane."""
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(7)
    k = 8
    lo = rng.uniform(-1.0, 0.5, (k, 2))
    hi = lo + rng.uniform(0.1, 0.8, (k, 2))
    quads = []
    for j in range(k):
        (a, b), (c, d) = lo[j], hi[j]
        quads += [[(a, b), (c, b), (c, d)], [(a, b), (c, d), (a, d)]]
    flat = np.repeat(rng.choice([-0.5, 0.0, 0.25, 0.25], k), 2)[:, None, None]
    tri = np.concatenate([np.broadcast_to(flat, (2 * k, 3, 1)), np.asarray(quads)], 2)
    v = (np.roll(tri, axis, axis=2).reshape(-1, 3) + offset).astype(np.float32)
    n = len(v) // 3
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1))
    m = data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])
    g, o = crt.Scene(m), OracleScene(m)
    count = 6_000
    t = v.reshape(-1, 3, 3).astype(np.float64)[rng.integers(0, n, count)]
    w = rng.dirichlet([0.5, 0.5, 0.5], count) * (rng.random((count, 3)) < 0.8)  # faces, edges and corners
    w[w.sum(1) == 0] = (1.0, 0.0, 0.0)
    p = np.einsum("ij,ijk->ik", w / w.sum(1, keepdims=True), t)
    d = rng.normal(size=(count, 3))
    d[: count // 4] *= np.array([1e-4, 1.0, 1.0])[[(c - axis) % 3 for c in range(3)]]  # grazing
    d[count // 4: count // 3] = np.eye(3)[rng.integers(0, 3, count // 3 - count // 4)]  # along an axis
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.hstack([p - d * rng.uniform(0.0, 3.0, (count, 1)), d])
    for any_hit in (False, True):
        gi, gt = g.trace(rays, any_hit=any_hit)
        oi, ot, _ = o.trace(rays, any_hit=any_hit)
        assert_equal(gi, oi, f"ids any={any_hit}")
        assert_equal(gt, ot, f"t any={any_hit}")
    g.check()


def test_underflowing_products(cuda):
    """Rays that start within 1e-20 to 1e-38 of a vertex near the origin: the filters' products underflow."""
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(13)
    n = 60
    v = rng.normal(size=(n, 3, 3))
    v[:, 0] = rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-38, -20, (n, 1))  # every triangle has a vertex there
    v = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1))
    m = data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])
    g, o = crt.Scene(m), OracleScene(m)
    count = 4_000
    start = rng.normal(size=(count, 3)) * 10.0 ** rng.uniform(-38, -20, (count, 1))
    d = rng.normal(size=(count, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.hstack([start - d * np.where(rng.random((count, 1)) < 0.5, 0.0, 1.0), d])
    for any_hit in (False, True):
        gi, gt = g.trace(rays, any_hit=any_hit)
        oi, ot, _ = o.trace(rays, any_hit=any_hit)
        assert_equal(gi, oi, f"ids any={any_hit}")
        assert_equal(gt, ot, f"t any={any_hit}")
    g.check()
