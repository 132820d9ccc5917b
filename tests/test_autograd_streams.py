"""The differentiable renderer on torch streams other than the default one: every call of a step takes that step's
inputs, whatever is still queued from the steps before."""
from types import SimpleNamespace

import numpy as np
import pytest


class _QueuedScene:
    """A scene whose default stream lags behind: what is issued there reads its arguments at the end, what is issued on
    torch's current stream reads them in turn with torch's own operations (on the CPU, at once)."""

    def __init__(self, current):
        self.current, self.late, self.verts, self.mats = current, [], [], []

    def _issue(self, into, x, stream):
        if getattr(stream, "cuda_stream", stream) == self.current:
            into.append(x.detach().clone())
        else:
            slot = len(into)
            into.append(None)
            self.late.append(lambda: into.__setitem__(slot, x.detach().clone()))

    def set_vertices(self, verts, rebuild, stream=None):
        self._issue(self.verts, verts, stream)

    def set_materials(self, mats, stream=None):
        self._issue(self.mats, mats, stream)


def test_inputs_are_ordered_with_the_current_stream(monkeypatch):
    torch = pytest.importorskip("torch")
    from crt import autograd, data
    nop = lambda *a: None  # noqa: E731
    stream, default = (SimpleNamespace(cuda_stream=k, synchronize=nop, wait_stream=nop) for k in (7, 0))
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: stream)
    monkeypatch.setattr(torch.cuda, "default_stream", lambda *a: default)
    r = object.__new__(autograd.Renderer)
    r.scene, r.mats, r.light = _QueuedScene(7), torch.zeros(5, 16, dtype=torch.float64), data.Light()
    verts, light = torch.zeros(3, 3), torch.zeros(3)
    for step in range(3):
        verts.fill_(step)
        r.set_inputs(verts, light, torch.full((5, 3), 1.0 + step, dtype=torch.float64))
    for read in r.scene.late:
        read()
    for step in range(3):
        assert (r.scene.mats[step][:, 3:6] == 1.0 + step).all(), f"materials of step {step}"
        assert (r.scene.verts[step] == step).all(), f"vertices of step {step}"


@pytest.mark.gpu
@pytest.mark.parametrize("switch", [False, True])
def test_steps_on_side_streams(cuda, switch):
    """Forwards without a wait between them, each with its own vertices and albedo, on one side stream or on two in
    turn (each waiting for the other's work): the images and gradients of the default stream."""
    torch = cuda
    from crt import autograd, data
    w = h = 48
    sc = data.config4(width=w, height=h, spp=2)
    r = autograd.Renderer(sc.mesh, sc.camera, sc.light, w, h, 2)
    light = torch.tensor(sc.light.position, dtype=torch.float64, device="cuda")
    steps = [(torch.from_numpy(np.asarray(sc.mesh.verts, np.float32)).cuda() + 0.01 * k,
              torch.full((sc.mesh.materials.shape[0], 3), 0.1 + 0.2 * k, dtype=torch.float64, device="cuda"))
             for k in range(4)]
    want = [[x.clone() for x in autograd.render(v, light, a, r)] for v, a in steps]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2 if switch else 1)]
    got = []
    for k, (v, a) in enumerate(steps):
        s = streams[k % len(streams)]
        s.wait_stream(streams[(k - 1) % len(streams)])
        with torch.cuda.stream(s):
            got.append(autograd.render(v * 1.0, light, a * 1.0, r))  # (temporaries of this stream)
    torch.cuda.synchronize()
    for k in range(4):
        assert torch.equal(got[k][0], want[k][0]), f"image of step {k}"
        assert torch.equal(got[k][1], want[k][1]), f"depth of step {k}"
    # one whole step, forward and backward
    grads = []
    for s in (torch.cuda.default_stream(), streams[0]):
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            v, a = (x.clone().requires_grad_() for x in steps[2])
            img, depth = autograd.render(v, light, a, r)
            grads.append(torch.autograd.grad((img ** 2).sum() + 0.1 * depth.sum(), (v, a)))
        torch.cuda.synchronize()
    for x, y in zip(*grads):  # (summed by atomics: the order varies)
        assert x.abs().sum() > 0
        assert torch.allclose(x, y, rtol=1e-6, atol=1e-9 * float(x.abs().max()))
