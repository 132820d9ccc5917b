"""Images of few pixels take more lanes per pixel and tiles of fewer pixels, and the widest ones another register
split: every split has to give the image of the others and of the oracle, sample by sample."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


def _soup(n, seed):
    from crt import data
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    v = (c + rng.normal(0.0, 0.08, (n, 3, 3)) + np.array([0.0, 0.0, -3.0])).reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    nrm = np.tile(np.array([[0.0, 0.6, 0.8]], np.float32), (3 * n, 1))
    return data.Mesh(v, idx, nrm, idx.copy(), np.zeros(n, np.int32), data.lambert_material()[None])


@pytest.mark.parametrize("w,h", [(1, 1), (3, 5), (64, 48), (97, 61), (150, 103)])
@pytest.mark.parametrize("spp", [1, 3, 8, 16, 37])
def test_small_images(cuda, w, h, spp):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    m = _soup(400, 11)
    cam, light = data.Camera(fov=60.0, focal_point=3.0, fstop=4.0), data.Light(position=(2.5, 2.5, -0.5), radius=0.4)
    g, o = crt.Scene(m), OracleScene(m)
    got = g.render(cam, light, w, h, spp, aux=True, rays=True, rgbd=True)
    ref = o.render(cam, light, w, h, spp=spp, aux=True, rays_in=got["rays"])
    assert_equal(got["hit_id"], ref["hit_id"], "hit ids")
    assert_equal(got["hit_t"], ref["hit_t"], "hit t")
    assert_equal(got["rgb8"], ref["rgb"], "image")
    plain = g.render(cam, light, w, h, spp, aux=True, rgbd=True)
    rec = g.render_recursive(cam, light, w, h, spp, 0)
    for k in ("rgb8", "rgb_f64", "depth", "hit_id", "hit_t", "shadow", "shadow_id"):
        assert_equal(plain[k], got[k], k)
    assert_equal(rec["rgb8"], got["rgb8"], "depth-0 recursive image")
    g.check()


@pytest.mark.parametrize("w,h,spp", [(640, 240, 1), (640, 240, 16), (450, 333, 4), (1201, 301, 2)])
def test_bands_match_the_image(cuda, w, h, spp):
    """A frame and its bands of rows: the bands are small images, the frame is not."""
    import crt
    from crt import data
    m, optics = data.optics_scene(nu=8, specular=True)
    cam, light = data.Camera(fov=60.0, focal_point=3.0, fstop=8.0), data.Light(position=(2.5, 2.5, -0.5), radius=0.4)
    g = crt.Scene(m)
    whole = g.render(cam, light, w, h, spp)["rgb8"].reshape(h, w, 3)
    deep = g.render_recursive(cam, light, w, h, min(spp, 4), 2, optics=optics)["rgb8"].reshape(h, w, 3)
    for r0, r1 in [(0, 1), (7, 30), (100, 140), (h - 3, h)]:
        band = g.render(cam, light, w, h, spp, rows=(r0, r1))["rgb8"].reshape(h, w, 3)
        assert_equal(band[h - r1:h - r0], whole[h - r1:h - r0], f"rows {r0}..{r1}")
        band = g.render_recursive(cam, light, w, h, min(spp, 4), 2, optics=optics, rows=(r0, r1))["rgb8"]
        assert_equal(band.reshape(h, w, 3)[h - r1:h - r0], deep[h - r1:h - r0], f"recursive rows {r0}..{r1}")
    g.check()
