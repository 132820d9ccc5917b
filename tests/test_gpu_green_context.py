"""Sorts and builds where the whole device is not to be had at once: on a stream of a green context that holds a part
of the SMs, which the cooperative sort's blocks would not fit; and captured into a graph, where they would."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import assert_equal

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def green(cuda, tmp_path_factory):
    from crt import build as b
    so = str(tmp_path_factory.mktemp("green") / "green_stream.so")
    subprocess.check_call([b.nvcc(), *b.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                           os.path.join(HERE, "probes", "green_stream.cu"), "-o", so, "-lcuda"])
    lib = ctypes.CDLL(so)
    stream, sms = ctypes.c_void_p(), ctypes.c_uint()
    if lib.green_stream_create(16, ctypes.byref(stream), ctypes.byref(sms)) != 0:
        pytest.skip("no green contexts here")
    assert sms.value < cuda.cuda.get_device_properties(0).multi_processor_count
    yield stream.value
    assert lib.green_stream_destroy() == 0


@pytest.mark.parametrize("n", [1024, 1025, 16385, 100_000, 1_000_003])
@pytest.mark.parametrize("bits", [16, 32])
def test_sort(cuda, green, n, bits):
    import crt
    torch = cuda
    k = torch.from_numpy(np.random.default_rng(n).integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
                         .view(np.int32)).cuda()
    ko, vo = torch.empty_like(k), torch.empty_like(k)
    torch.cuda.synchronize()
    crt.sort_pairs(k, None, ko, vo, key_bits=bits, stream=green)
    keys = k.cpu().numpy().view(np.uint32)
    order = np.argsort(keys, kind="stable")
    assert_equal(ko.cpu().numpy().view(np.uint32), keys[order], "keys")
    assert_equal(vo.cpu().numpy(), order.astype(np.int32), "values")


@pytest.mark.parametrize("n", [2000, 32768, 60_000])
def test_build(cuda, green, n):
    import crt
    from crt import data
    m = data.soup(n, seed=n)
    want = crt.Scene(m).export()
    s = crt.Scene(m, stream=green)
    s.build(stream=green)
    s.check(stream=green)
    got = s.export()
    for k in ("codes", "ids", "nodes", "node_boxes"):
        assert_equal(got[k], want[k], k)


def test_captured_build(cuda):
    import crt
    from crt import data
    torch = cuda
    m = data.soup(40_000, seed=3)
    s = crt.Scene(m)
    want = s.export()
    g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=side):
        s.build(stream=side)
    s.set_vertices(np.ascontiguousarray(m.verts[::-1]), rebuild=True)
    s.set_vertices(m.verts, rebuild=False)
    g.replay()
    torch.cuda.synchronize()
    s.check()
    got = s.export()
    for k in ("codes", "ids", "nodes", "node_boxes"):
        assert_equal(got[k], want[k], k)
