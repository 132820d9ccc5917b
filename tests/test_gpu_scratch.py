"""The memory that calls keep between them: it is bounded whichever contexts the calls come from, stays while a scene
is alive, and goes back with the last scene or on request.  Each test is a process of its own, for the free memory to
be its alone."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PRELUDE = """
import ctypes, sys
sys.path.insert(0, {pkg!r})
import numpy as np
import torch
import crt
from crt import data
MB = 1 << 20
N = 8_000_000  # 64 MB of keys and values alone
torch.cuda.set_device(0)
a = torch.arange(N, dtype=torch.int32, device="cuda")
b, c = torch.empty_like(a), torch.empty_like(a)
def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
def sort(x=a, y=b, z=c):
    ptr = [ctypes.c_void_p(t.data_ptr() if hasattr(t, "data_ptr") else t) for t in (x, y, z)]
    assert crt.lib().crt_sort_pairs(ptr[0], None, ptr[1], ptr[2], N, 32, None) == 0
crt.sort_pairs(a[:4096], None, b[:4096], c[:4096])  # the kernels are loaded
"""


def _run(body):
    code = PRELUDE.format(pkg=os.path.join(ROOT, "cuda-rt_gb300")) + body
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_sorts_alone(cuda):
    _run("""
crt.lib().crt_scene_destroy(None)
before = free()
sort()
kept = before - free()
assert 32 * MB < kept <= 288 * MB, kept
for _ in range(3):
    sort()
assert before - free() == kept
crt.lib().crt_scene_destroy(None)
assert before - free() < 8 * MB
sort()
assert torch.equal(b, a) and torch.equal(c, a)
""")


def test_scenes_hold_the_memory(cuda):
    _run("""
scenes = [crt.Scene(data.config0(n=500).mesh) for _ in range(2)]
before = free()
sort()
kept = before - free()
assert kept > 32 * MB, kept
crt.lib().crt_scene_destroy(None)
scenes.pop().close()
assert before - free() > 32 * MB  # the other scene's calls go on using it
scenes.pop().close()
assert before - free() < 8 * MB
""")


def test_alternating_contexts(cuda):
    _run("""
cu = ctypes.CDLL("libcuda.so.1")
def ok(rc):
    assert rc == 0, rc
ctx, old = ctypes.c_void_p(), ctypes.c_void_p()
ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0))  # now the current one
ptrs = []
for _ in range(3):
    p = ctypes.c_uint64()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(4 * N)))
    ok(cu.cuMemcpy(p, ctypes.c_uint64(a.data_ptr()), ctypes.c_size_t(4 * N)))
    ptrs.append(p.value)
sort(*ptrs)  # the kernels are loaded here too
ok(cu.cuCtxPopCurrent_v2(ctypes.byref(old)))
sort()
assert torch.equal(b, a) and torch.equal(c, a)  # (what this takes is no part of the measure either)
before = free()
for _ in range(6):
    ok(cu.cuCtxPushCurrent_v2(ctx))
    sort(*ptrs)
    ok(cu.cuCtxPopCurrent_v2(ctypes.byref(old)))
    sort()
    assert torch.equal(b, a) and torch.equal(c, a)
assert before - free() < 64 * MB, (before - free()) / MB
""")
