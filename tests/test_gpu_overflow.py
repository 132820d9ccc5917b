"""Scenes and rays so large that the FP32 triangle filters' products overflow while the exact test's do not: the hits
must be the oracle's."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 600])
@pytest.mark.parametrize("spread", [0.05, 0.5])
@pytest.mark.parametrize("scale,length", [(1e18, 1.0), (1e19, 1.0), (2e19, 1.0), (4e19, 1.0), (1e20, 1.0), (1e21, 1.0),
                                          (1e30, 1.0), (1e12, 1e16), (1e10, 1e19), (3e9, 1e20), (1.0, 1e36)])
def test_large_products(cuda, scale, length, spread, n):
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    rng = np.random.default_rng(n)
    v = (rng.uniform(-1.0, 1.0, (n, 1, 3)) + rng.normal(0.0, spread, (n, 3, 3))) * scale
    v = v.reshape(-1, 3).astype(np.float32)
    idx = np.arange(3 * n, dtype=np.int32).reshape(n, 3)
    m = data.Mesh(v, idx, np.tile(np.array([[0.0, 0.0, 1.0]], np.float32), (3 * n, 1)), idx.copy(),
                  np.zeros(n, np.int32), data.lambert_material()[None])
    g, o = crt.Scene(m), OracleScene(m)
    count = 600
    lo, hi = v.astype(np.float64).min(0), v.astype(np.float64).max(0)
    org = rng.uniform(lo - 0.1 * (hi - lo), hi + 0.1 * (hi - lo), (count, 3))
    d = v.astype(np.float64)[idx[rng.integers(0, n, count)]].mean(1) - org
    d *= length / np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.hstack([org, d])
    for any_hit in (False, True):
        gi, gt = g.trace(rays, any_hit=any_hit)
        oi, ot, _ = o.trace(rays, any_hit=any_hit)
        assert (oi >= 0).any() or scale / length < 1e-8  # (|t| < 1e-8 is no hit)
        assert_equal(gi, oi, f"ids any={any_hit}")
        assert_equal(gt, ot, f"t any={any_hit}")
    g.check()
