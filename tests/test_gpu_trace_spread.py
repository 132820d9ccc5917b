"""Batched rays at every number of rays a warp can own (one for few rays, up to 32), the last chunk ragged: each ray bit
for bit as the oracle's."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per", [1, 2, 4, 8, 16, 32])
@pytest.mark.parametrize("any_hit", [False, True])
def test_rays_per_warp(cuda, per, any_hit):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    m = data.soup(3000, seed=4, sigma=0.05)
    g, o = crt.Scene(m), OracleScene(m)
    warps = cuda.cuda.get_device_properties(0).multi_processor_count * 8 * 4  # resident: eight blocks of four per SM
    n = per * warps + per // 2 + 1  # as many chunks as warps and one more, not a full one when per > 1
    rng = np.random.default_rng(per)
    d = rng.normal(size=(n, 3))
    rays = np.hstack([np.array([0.0, 0.0, -3.0]) + rng.uniform(-1.5, 1.5, (n, 3)),
                      d / np.linalg.norm(d, axis=1, keepdims=True)])
    for k in (n, per * warps - per // 2):  # (one chunk fewer)
        gi, gt = g.trace(rays[:k], any_hit=any_hit)
        oi, ot, _ = o.trace(rays[:k], any_hit=any_hit)
        assert_equal(gi, oi, "ids")
        assert_equal(gt, ot, "t")
    g.check()
