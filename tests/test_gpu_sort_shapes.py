"""The standalone sort around the sizes where its kernel changes shape (one block, the fewest items per thread that
leave no more tiles than SMs, the look-back passes beyond), with one to four passes: keys and values must be those of
a stable sort."""
import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu

SIZES = [1024, 1025, 2047, 16384, 152 * 1024, 152 * 1024 + 1, 304 * 1024 + 1, 608 * 1024 + 1, 1064 * 1024 + 1,
         1216 * 1024 + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits,spread", [(10, 1 << 10), (20, 37), (30, 1 << 30), (32, 1 << 32)])
def test_sort_shapes(cuda, n, bits, spread):
    import torch

    import crt
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, spread, n, dtype=np.uint64).astype(np.uint32)
    v = rng.integers(0, 1 << 31, n, dtype=np.int64).astype(np.int32)
    order = np.argsort(k, kind="stable")
    kd, vd = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v).cuda()
    for vals, want in ((vd, v[order]), (None, order.astype(np.int32))):
        ko, vo = torch.empty_like(kd), torch.empty_like(kd)
        crt.sort_pairs(kd, vals, ko, vo, key_bits=bits)
        assert_equal(ko.cpu().numpy().view(np.uint32), k[order], "keys")
        assert_equal(vo.cpu().numpy(), want, "values")
    assert_equal(kd.cpu().numpy().view(np.uint32), k, "input keys")
    if n <= crt.SORT_NOALLOC_MAX_PAIRS:
        crt.sort_pairs_noalloc(kd, vd, ko, vo, key_bits=bits)
        assert_equal(vo.cpu().numpy(), v[order], "values, no allocation")


@pytest.mark.parametrize("n", [1025, 8192, 152 * 1024, 152 * 4096 + 1, 152 * 8192 - 5])
@pytest.mark.parametrize("kind", ["equal", "two", "last tile"])
def test_skewed_digits(cuda, n, kind):
    """One digit holding whole tiles (the largest 16-bit counts), two digits, and a digit of the last tile alone."""
    import torch
    import crt
    k = torch.full((n,), 0x2AA55AA5, dtype=torch.int32, device="cuda")
    if kind == "two":
        k[torch.arange(n, device="cuda") % 3 == 1] = 0x15455AA5
    elif kind == "last tile":
        k[-700:] = 0x00100400
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    crt.sort_pairs(k, v, ko, vo, key_bits=30)
    ks, ix = torch.sort(k, stable=True)
    assert torch.equal(ko, ks)
    assert torch.equal(vo, v[ix])


@pytest.mark.parametrize("n", [16384, 32767, 32768, 32769])
def test_builds_beside_the_cooperative_sort(cuda, n):
    """Builds on both sides of the size from which their sort is one cooperative launch."""
    import crt
    from crt import data
    from oracle.oracle import OracleScene
    m = data.soup(n, seed=n)
    ge, oe = crt.Scene(m).export(), OracleScene(m).export()
    for k in ("codes", "ids", "nodes", "node_boxes"):
        assert_equal(ge[k], oe[k], k)
