"""The beam test that drops blocks of pixels no camera ray of which can hit anything: whole images and every
auxiliary output must equal the oracle's (which has no such test), whatever the lens, the focus, the side of the
camera the mesh is on and the size of the image."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


def _cluster(n, centre, size, seed):
    from crt import data
    rng = np.random.default_rng(seed)
    c = np.asarray(centre) + rng.uniform(-size, size, (n, 1, 3))
    v = (c + rng.normal(0.0, 0.1 * size, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.6, 0.8]], np.float32), (3 * n, 1))
    return data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])


@pytest.mark.parametrize("fstop,focal", [(np.inf, 1.0), (10.0, 3.0), (0.5, 3.0), (2.0, 0.2), (4.0, -3.0), (4.0, 1e-9)])
@pytest.mark.parametrize("centre,size", [((0, 0, -3), 0.2), ((0.9, -0.5, -3), 0.1), ((0.3, 0.2, 2.0), 0.2),
                                         ((0, 0, 0), 0.5), ((2.0, 0, -3), 0.05), ((0, 0, -400), 20.0)])
@pytest.mark.parametrize("w,h,spp", [(67, 45, 4), (40, 33, 1)])
def test_beam_keeps_images(cuda, fstop, focal, centre, size, w, h, spp):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    m = _cluster(300, centre, size, 5)
    cam = data.Camera(fov=60.0, focal_point=focal, fstop=fstop)
    light = data.Light(position=(2.5, 2.5, -0.5))
    g, o = crt.Scene(m), OracleScene(m)
    with_rays = g.render(cam, light, w, h, spp, aux=True, rays=True, rgbd=True)  # rays asked for: no block is dropped
    got = g.render(cam, light, w, h, spp, aux=True, rgbd=True)
    for k in ("rgb8", "rgb_f64", "depth", "hit_id", "hit_t", "shadow", "shadow_id"):
        assert_equal(got[k], with_rays[k], k)
    ref = o.render(cam, light, w, h, spp=spp, aux=True, rays_in=with_rays["rays"])
    assert_equal(got["hit_id"], ref["hit_id"], "hit ids")
    assert_equal(got["rgb8"], ref["rgb"], "image")
    r0 = g.render_recursive(cam, light, w, h, spp, 0)
    assert_equal(r0["rgb8"], got["rgb8"], "depth-0 recursive image")
    assert_equal(r0["hit_t"], got["hit_t"], "depth-0 recursive t")
    rows = g.render(cam, light, w, h, spp, rows=(8, 31))["rgb8"].reshape(h, w, 3)[h - 31:h - 8]
    assert_equal(rows, got["rgb8"].reshape(h, w, 3)[h - 31:h - 8], "a band of rows")
    g.check()
