"""Performance cases: what programs built on this library ask of it.

A case is a dict of plain values.  Five kinds of call are covered, each
through the Python front end over the C ABI:

  frame      a mesh update (full LBVH build, rebuild from new vertices, refit,
             or none) and a rendered image
  recursive  an image with reflected and refracted rays
  batch      many meshes built and rendered together
  diff       one differentiable step: image, depth and the gradients
  trace      ray queries, with or without an update of the mesh before them
  sort       the stable key/value sort

Sizes are those of the repository's own configurations (crt.data.config0-4,
bench.py, the command-line renderer's defaults, the smoke test) and of its
tests, and `draw` spreads over the ranges between them.  Inputs come from the
seed alone: another seed is another displaced sphere, soup, set of rays or
keys.  Images are compared as 8-bit pixels and hits as triangle ids, both
whole numbers; `exact` gives distances and gradients in 64 bits by brute
force over all triangles.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "cuda-rt_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "cuda-rt_gb300"))

import crt  # noqa: E402
from crt import autograd, data  # noqa: E402

DEV = "cuda"
CAM_POS = (0.0, 0.0, -3.0)
EYE_DEPTH = -3.0  # the meshes sit at (0, 0, -3) in the camera's frame


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest image: a preview or a test render, where launches and host calls count.
        dict(name="frame_tiny", kind="frame", mesh="soup", n=2000, update="build", width=64, height=48, spp=2,
             lens=False, shade="point", host=False),
        # The plain method's small configuration: 100k triangles, one sample per pixel, pinhole.
        dict(name="frame_small", kind="frame", mesh="soup", n=100_000, update="rebuild", width=640, height=480, spp=1,
             lens=False, shade="point", host=False),
        # The plain method's large configuration, which bench.py times: 1,003,520 triangles, thin lens.
        dict(name="frame_large", kind="frame", mesh="sphere", n=224, update="build", width=1920, height=1080, spp=16,
             lens=True, shade="point", host=False),
        # One frame of an animation that keeps its topology: new vertices, refit, image.
        dict(name="frame_refit", kind="frame", mesh="sphere", n=224, update="refit", width=1280, height=720, spp=4,
             lens=True, shade="point", host=False),
        # What the command-line renderer does by default (512 x 512, 20 samples, thin lens, area light with
        # falloff, highlights), the image pulled into host memory.
        dict(name="image_host", kind="frame", mesh="sphere", n=60, update="none", width=512, height=512, spp=20,
             lens=True, shade="full", host=True),
        # Mirror and glass, three levels deep.
        dict(name="recursive", kind="recursive", n=64, width=1280, height=720, spp=4, depth=3),
        # Meshes of very different sizes built and rendered in one go (a data generator's step).
        dict(name="batch", kind="batch", count=24, lo=1000, hi=500_000, width=256, height=256, spp=4),
        # One optimisation step over vertices, light and a per-triangle albedo.
        dict(name="diff_step", kind="diff", n=100, width=512, height=512, spp=4),
        # Incoherent closest-hit queries (collision checks, sampling) against a soup, in device memory.
        dict(name="trace_closest", kind="trace", mesh="soup", n=100_000, update="none", rays=1_000_000,
             pattern="random", any_hit=False),
        # Visibility queries: occlusion rays from points of a surface, a ragged number of them.
        dict(name="trace_any", kind="trace", mesh="sphere", n=100, update="none", rays=262_147, pattern="surface",
             any_hit=True),
        # A simulation step: the mesh moved, the tree rebuilt, a few thousand rays cast.
        dict(name="rebuild_probe", kind="trace", mesh="sphere", n=31, update="rebuild", rays=4096, pattern="camera",
             any_hit=False),
        # The sort by itself, on 32-bit keys.
        dict(name="sort", kind="sort", n=1_000_003, bits=32, values=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "recursive", "batch", "diff", "trace", "trace", "trace", "sort"])
    if kind == "frame":
        mesh = rng.choice(["soup", "sphere"])
        w = _log(rng, 48, 1920)
        h = max(32, min(1080, int(w * rng.uniform(0.5, 1.0))))
        # at most the samples of the large configuration; a soup costs several times a sphere's rays
        spp = min(rng.choice([1, 2, 3, 4, 8, 16, 20]), max(1, 33_177_600 // (w * h) // (8 if mesh == "soup" else 1)))
        return dict(kind="frame", mesh=mesh, n=_log(rng, 300, 200_000) if mesh == "soup" else _log(rng, 5, 224),
                    update=rng.choice(["build", "rebuild", "refit", "none"]), width=w, height=h, spp=spp,
                    lens=rng.random() < 0.6, shade=rng.choice(["point", "point", "full"]), host=rng.random() < 0.3)
    if kind == "recursive":
        w = _log(rng, 64, 1280)
        return dict(kind="recursive", n=_log(rng, 6, 64), width=w, height=max(48, int(w * 0.5625)),
                    spp=rng.choice([1, 2, 3, 4]), depth=rng.choice([1, 2, 3]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(2, 24), lo=rng.choice([1, 100, 1000]),
                    hi=_log(rng, 5000, 500_000), width=_log(rng, 32, 256), height=_log(rng, 32, 256),
                    spp=rng.choice([1, 2, 3, 4]))
    if kind == "diff":
        return dict(kind="diff", n=_log(rng, 10, 100), width=_log(rng, 33, 512), height=_log(rng, 33, 512),
                    spp=rng.choice([1, 2, 3, 4]))
    if kind == "trace":
        mesh = rng.choice(["soup", "sphere"])
        return dict(kind="trace", mesh=mesh, n=_log(rng, 300, 200_000) if mesh == "soup" else _log(rng, 5, 224),
                    update=rng.choice(["none", "none", "rebuild", "refit"]), rays=_log(rng, 100, 1_000_000),
                    pattern=rng.choice(["random", "surface", "camera"]), any_hit=rng.random() < 0.4)
    return dict(kind="sort", n=_log(rng, 1000, 4_000_000), bits=rng.choice([16, 30, 32]), values=rng.random() < 0.7)


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed & 0x7FFFFFFF)
    return g


@functools.lru_cache(maxsize=4)
def _unit_sphere(nu):
    """Vertices (unit directions, float64) and faces of the geodesic sphere."""
    m = data.icosphere(nu, amp=0.0)
    v = torch.from_numpy(m.verts.astype(np.float64)).to(DEV)
    v[:, 2] -= EYE_DEPTH
    return v / v.norm(dim=1, keepdim=True), torch.from_numpy(m.vidx).to(DEV)


def _waves(g, u, amp, k=4):
    """A smooth displacement of the unit sphere: amp * sum of k random sine waves."""
    f = torch.rand(k, generator=g, device=DEV, dtype=torch.float64) * 7 + 1
    ph = torch.rand(k, generator=g, device=DEV, dtype=torch.float64) * (2 * math.pi)
    ax = torch.randn(k, 3, generator=g, device=DEV, dtype=torch.float64)
    ax = ax / ax.norm(dim=1, keepdim=True)
    return amp * torch.sin((u @ ax.T) * f + ph).sum(1, keepdim=True)


def _materials(shade):
    m = np.zeros((1, 16))
    m[0, 3:6] = 0.8 if shade != "full" else (0.7, 0.6, 0.5)
    m[0, 15] = 20.0
    if shade == "full":
        m[0, 6:9] = 0.3
    return m


def _mesh(case, seed, shade="point"):
    """A mesh in device memory and a second set of vertices with the same topology."""
    g = _gen(seed)
    if case["mesh"] == "sphere":
        u, faces = _unit_sphere(case["n"])
        v = u * (1.0 + _waves(g, u, 0.05))
        a, b, c = (v[faces[:, k].long()] for k in range(3))
        fn = torch.linalg.cross(b - a, c - a)
        nrm = torch.zeros_like(v)
        for k in range(3):
            nrm.index_add_(0, faces[:, k].long(), fn)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
        moved = v + 0.02 * torch.sin(0.7 + 5.0 * v[:, :1]) * nrm
        vidx = faces.contiguous()
    else:
        n = case["n"]
        cent = torch.rand(n, 1, 3, generator=g, device=DEV, dtype=torch.float64) * 2 - 1
        v = cent + 0.01 * torch.randn(n, 3, 3, generator=g, device=DEV, dtype=torch.float64)
        moved = (v + 0.02 * torch.sin(3.0 * cent)).reshape(-1, 3)
        fn = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        nrm = (fn / fn.norm(dim=1, keepdim=True)).repeat_interleave(3, 0)
        v = v.reshape(-1, 3)
        vidx = torch.arange(3 * n, device=DEV, dtype=torch.int32).reshape(n, 3)
    shift = torch.tensor([0.0, 0.0, EYE_DEPTH], device=DEV, dtype=torch.float64)
    verts, moved = (v + shift).float().contiguous(), (moved + shift).float().contiguous()
    m = data.Mesh(verts, vidx, nrm.float().contiguous(), vidx,
                  torch.zeros(vidx.shape[0], device=DEV, dtype=torch.int32), _materials(shade))
    return m, moved


def _light(shade):
    if shade == "full":  # the command-line renderer's light, moved to where it lights the mesh
        return data.Light(position=(2.5, 2.5, 0.5), radius=0.5, constant_term=0.0, linear_term=0.1,
                          quadratic_term=0.01)
    return data.Light(position=data.light_for((2.0, 2.0, -2.0), CAM_POS))


def _rays(case, seed, mesh):
    g = _gen(seed + 7919)
    n = case["rays"]
    centre = torch.tensor([0.0, 0.0, EYE_DEPTH], device=DEV, dtype=torch.float64)
    rnd = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)  # noqa: E731
    if case["pattern"] == "random":
        o = centre + (rnd(n, 3) * 2 - 1) * 1.5
        d = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    elif case["pattern"] == "surface":
        # from points just above the surface into the outer half space, neighbours next to each other
        f = torch.sort(torch.randint(0, mesh.vidx.shape[0], (n,), generator=g, device=DEV))[0]
        tri = mesh.verts.double()[mesh.vidx[f].long()]
        w = rnd(n, 3) + 0.05
        w = w / w.sum(1, keepdim=True)
        nrm = mesh.normals.double()[mesh.nidx[f].long()].mean(1)
        o = (tri * w[:, :, None]).sum(1) + 1e-4 * nrm
        d = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
        d = torch.where((d * nrm).sum(1, keepdim=True) < 0, -d, d)
    else:  # a raster of view rays from a point in front of the mesh
        w = max(1, int(math.sqrt(n)))
        i = torch.arange(n, device=DEV)
        x = ((i % w) + rnd(n)) / w - 0.5
        y = (torch.div(i, w, rounding_mode="floor") + rnd(n)) / max(1, n // w) - 0.5
        o = torch.zeros(n, 3, device=DEV, dtype=torch.float64)
        d = torch.stack([x, y, torch.full_like(x, -1.2)], 1)
    d = d / d.norm(dim=1, keepdim=True)
    return torch.cat([o, d], 1).contiguous()


# ------------------------------------------------------------------ states
def prepare(case, seed):
    k = case["kind"]
    s = dict(case=case)
    if k == "frame":
        mesh, moved = _mesh(case, seed, case["shade"])
        s["scene"] = crt.Scene(mesh)
        s["verts"] = [mesh.verts, moved]
        s["turn"] = 0
        s["camera"] = data.Camera(fov=60.0, focal_point=3.0, fstop=10.0 if case["lens"] else math.inf)
        s["light"] = _light(case["shade"])
        if not case["host"]:
            s["out"] = dict(rgb8=torch.empty((case["width"] * case["height"], 3), dtype=torch.uint8, device=DEV))
    elif k == "recursive":
        mesh, optics = data.optics_scene(nu=case["n"], specular=True)
        g = np.random.default_rng(seed)
        optics[1, :3] = g.uniform(0.6, 0.9)
        optics[2, 3] = g.uniform(1.3, 1.7)
        off = g.uniform(-0.05, 0.05, 3).astype(np.float32)
        mesh.verts = mesh.verts + off
        s["scene"] = crt.Scene(mesh)
        s["optics"] = torch.from_numpy(optics).to(DEV)
        s["camera"] = data.Camera(fov=50.0, focal_point=3.0, fstop=25.0)
        s["light"] = data.Light(position=data.light_for((2.0, 2.5, -2.0), CAM_POS), radius=0.3, linear_term=0.02,
                                quadratic_term=0.01)
        s["out"] = dict(rgb8=torch.empty((case["width"] * case["height"], 3), dtype=torch.uint8, device=DEV))
    elif k == "batch":
        rng = np.random.default_rng(seed)
        sizes = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["count"])).astype(np.int64)
        sizes[0] = case["hi"]
        meshes, views = [], []
        for m in range(case["count"]):
            d = rng.normal(size=3)
            pos = tuple(4.0 * d / np.linalg.norm(d))
            meshes.append(data.soup(int(sizes[m]), scale=float(rng.uniform(0.5, 4.0)), cam_pos=pos, rng=rng))
            views.append((data.Camera(fov=60.0, focal_point=4.0, fstop=25.0),
                          data.Light(position=data.light_for(tuple(np.asarray(pos) * 0.5 + np.array([2.0, 2.0, 0.0])),
                                                             pos)), case["width"], case["height"], case["spp"]))
        s["batch"] = crt.Batch(meshes, views)
        s["batch"].autotune()
        s["image"] = torch.empty((int(s["batch"].offsets[-1]), 3), dtype=torch.uint8, device=DEV)
    elif k == "diff":
        m, moved = _mesh(dict(mesh="sphere", n=case["n"]), seed)
        g = _gen(seed + 31)
        n = m.vidx.shape[0]
        mats = np.zeros((n, 16))
        mats[:, 3:6] = 0.7
        host = data.Mesh(m.verts.cpu().numpy(), m.vidx.cpu().numpy(), m.normals.cpu().numpy(), m.nidx.cpu().numpy(),
                         np.arange(n, dtype=np.int32), mats)
        s["renderer"] = autograd.Renderer(host, data.Camera(fov=60.0), data.Light(), case["width"], case["height"],
                                          case["spp"])
        px = case["width"] * case["height"]
        s["verts"] = moved.clone().requires_grad_()
        s["light"] = torch.tensor(data.light_for((3.0, 3.0, -3.0), CAM_POS), dtype=torch.float64, device=DEV,
                                  requires_grad=True)
        s["albedo"] = (torch.rand(n, 3, generator=g, device=DEV, dtype=torch.float64) * 0.4 + 0.5).requires_grad_()
        s["grads"] = (torch.randn(px, 3, generator=g, device=DEV, dtype=torch.float64) / px,
                      0.1 * torch.randn(px, generator=g, device=DEV, dtype=torch.float64) / px)
        s["mesh"] = m
    elif k == "trace":
        mesh, moved = _mesh(case, seed)
        s["scene"] = crt.Scene(mesh)
        s["verts"] = moved
        s["rays"] = _rays(case, seed, mesh)
        s["mesh"] = mesh
    else:
        g = _gen(seed)
        n, bits = case["n"], case["bits"]
        keys = torch.randint(0, 1 << bits, (n,), generator=g, device=DEV, dtype=torch.int64)
        s["keys"] = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)  # the same 32 bits
        s["vals"] = torch.randint(0, 1 << 30, (n,), generator=g, device=DEV, dtype=torch.int32) if case["values"] \
            else None
        s["out"] = (torch.empty_like(s["keys"]), torch.empty_like(s["keys"]))
    return s


def run(s):
    c = s["case"]
    k = c["kind"]
    if k == "frame":
        sc = s["scene"]
        if c["update"] == "build":
            sc.build()
        elif c["update"] != "none":
            s["turn"] = 1 - s["turn"]  # an animation: other vertices each frame
            sc.set_vertices(s["verts"][s["turn"]], rebuild=c["update"] == "rebuild")
        return sc.render(s["camera"], s["light"], c["width"], c["height"], c["spp"], out=s.get("out"))["rgb8"]
    if k == "recursive":
        return s["scene"].render_recursive(s["camera"], s["light"], c["width"], c["height"], c["spp"], c["depth"],
                                           s["optics"], out=s["out"])["rgb8"]
    if k == "batch":
        return s["batch"].run(s["image"])
    if k == "diff":
        args = (s["verts"], s["light"], s["albedo"])
        img, depth = autograd.render(*args, s["renderer"])
        gv, gl, ga = torch.autograd.grad((img, depth), args, s["grads"])
        return dict(image=img.detach(), depth=depth.detach(), vertices=gv, light=gl, albedo=ga)
    if k == "trace":
        if c["update"] != "none":
            s["scene"].set_vertices(s["verts"], rebuild=c["update"] == "rebuild")
        ids, t = s["scene"].trace(s["rays"], any_hit=c["any_hit"])
        return dict(ids=ids, t=t)
    ko, vo = s["out"]
    crt.sort_pairs(s["keys"], s["vals"], ko, vo, key_bits=c["bits"])
    return dict(keys=ko, vals=vo)


# ------------------------------------------------------------------ work
def _tris(case):
    return 20 * case["n"] ** 2 if case.get("mesh", "sphere") == "sphere" else case["n"]


def _verts(case):
    return 10 * case["n"] ** 2 + 2 if case.get("mesh", "sphere") == "sphere" else 3 * case["n"]


def _per_ray(n):
    """One ray's unavoidable arithmetic: a path of four-wide boxes down to one triangle."""
    return 48.0 * max(1.0, math.log(max(n, 2), 4)) + 60.0


def work(case):
    k = case["kind"]
    if k == "sort":
        return dict(bytes=case["n"] * (8.0 * 2 if case["values"] else 12.0), flops=0.0)
    if k == "trace":
        n = _tris(case)
        built = 12.0 * _verts(case) if case["update"] != "none" else 0.0
        return dict(bytes=built + 12.0 * n + 12.0 * _verts(case) + case["rays"] * 60.0,
                    flops=case["rays"] * _per_ray(n))
    if k == "batch":
        tris = case["hi"] + (case["count"] - 1) * (case["hi"] - case["lo"]) / max(math.log(case["hi"] / case["lo"]),
                                                                                  1e-9)
        px = case["count"] * case["width"] * case["height"]
        return dict(bytes=tris * (36 + 12) + 3.0 * px, flops=px * case["spp"] * (80 + _per_ray(tris / case["count"])))
    px = case["width"] * case["height"]
    rays = float(px * case["spp"])
    if k == "recursive":
        n = 25 * case["n"] ** 2
        return dict(bytes=n * 36.0 + 3.0 * px, flops=2 * rays * (80 + _per_ray(n)))
    n = _tris(case)
    if k == "diff":
        # vertices, albedo and the gradients of image and depth in; image, depth and the three gradients out
        return dict(bytes=12.0 * _verts(case) * 2 + 24.0 * n * 2 + 12.0 * n + 32.0 * px * 2,
                    flops=rays * (200 + 2 * _per_ray(n)))
    return dict(bytes=12.0 * _verts(case) + 12.0 * n + 3.0 * px, flops=rays * (80 + _per_ray(n)))


# ------------------------------------------------------------------ 64-bit results
def _morton_order(verts, vidx):
    """The triangles in the order of their 30-bit Morton codes (ties by index)."""
    tri = verts[vidx.long()]
    lo, hi = tri.amin(1), tri.amax(1)
    mn, mx = lo.amin(0), hi.amax(0)
    q = (0.5 * (lo.double() + hi.double()) - mn.double()) / (mx.double() - mn.double())
    cell = (q * 1024.0).clamp(0.0, 1023.0).float().long()
    code = torch.zeros(len(vidx), dtype=torch.int64, device=DEV)
    for b in range(10):
        for a in range(3):
            code |= ((cell[:, a] >> b) & 1) << (3 * b + 2 - a)
    return torch.sort(code, stable=True)[1]


def _hits(verts, vidx, rays, any_hit):
    """Brute force: each ray against every triangle in Morton order, in 64 bits; (sorted position, t) of
    the least t, or of the first hit in that order; position -1 for a miss.  A ray's t may be negative,
    as the library's."""
    tri = verts.double()[vidx[_morton_order(verts, vidx)].long()]
    a, ab, ac = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = torch.linalg.cross
    nrm = cross(ac, ab)  # det = d . (ac x ab)
    # alpha's numerator (o - a).(d x ac) = (o x d).ac + d.(a x ac), beta's (o - a).(ab x d) alike
    an_w, bn_w = torch.cat([cross(a, ac), ac], 1), torch.cat([cross(ab, a), -ab], 1)
    tn_w = torch.cat([-nrm, (nrm * a).sum(1, keepdim=True)], 1)
    n = len(tri)
    best_t = torch.zeros(len(rays), dtype=torch.float64, device=DEV)
    best_k = torch.full((len(rays),), -1, dtype=torch.int64, device=DEV)
    step = max(1, 250_000_000 // n)
    for r0 in range(0, len(rays), step):
        o, d = rays[r0:r0 + step, :3], rays[r0:r0 + step, 3:]
        pl = torch.cat([d, cross(o, d)], 1)
        det = d @ nrm.T
        inv = 1.0 / det
        al = (pl @ an_w.T).mul_(inv)
        be = (pl @ bn_w.T).mul_(inv)
        ok = (det.float().abs() >= 1e-8) & (al >= 0) & (be >= 0)
        ok &= al.add_(be) <= 1
        del det, be
        t = (torch.cat([o, torch.ones_like(o[:, :1])], 1) @ tn_w.T).mul_(inv)
        ok &= t.float().abs() >= 1e-8
        if any_hit:
            k = ok.to(torch.uint8).argmax(1)  # the first of the largest
        else:
            k = torch.where(ok, t, math.inf).argmin(1)
        hit = ok.gather(1, k[:, None])[:, 0]
        best_k[r0:r0 + step] = torch.where(hit, k, -1)
        best_t[r0:r0 + step] = torch.where(hit, t.gather(1, k[:, None])[:, 0], 0.0)
    return best_k, best_t


def _exact_diff(case, s):
    """The pinhole image, depth and gradients: the hits by brute force, the rest by 64-bit autograd."""
    w, h = case["width"], case["height"]
    v32, m = s["verts"].detach(), s["mesh"]
    verts, light, albedo = (x.detach().double().clone().requires_grad_() for x in
                            (s["verts"], s["light"], s["albedo"]))
    ang = math.tan(math.pi * 0.5 * 60.0 / 180.0)
    px = (2 * ((torch.arange(w, device=DEV, dtype=torch.float64) + 0.5) / w) - 1) * ang * (w / h)
    py = (1 - 2 * ((torch.arange(h, device=DEV, dtype=torch.float64) + 0.5) / h)) * ang
    py = py.flip(0)  # the image is stored bottom row first
    d = torch.stack([px[None, :].expand(h, w), py[:, None].expand(h, w), torch.full((h, w), -1.0, device=DEV,
                                                                                   dtype=torch.float64)], 2)
    d = (d / d.norm(dim=2, keepdim=True)).reshape(-1, 3)
    order = _morton_order(v32, m.vidx)
    k, _ = _hits(v32, m.vidx, torch.cat([torch.zeros_like(d), d], 1), False)
    pix = torch.nonzero(k >= 0)[:, 0]
    f = order[k[pix]]
    d = d[pix]
    tri = verts[m.vidx[f].long()]
    a, ab, ac = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    cross = torch.linalg.cross
    p = cross(d, ac)
    det = (ab * p).sum(1)
    al = (-a * p).sum(1) / det
    q_ = cross(-a, ab)
    be = (d * q_).sum(1) / det
    t = (ac * q_).sum(1) / det
    nr = m.normals.double()[m.nidx[f].long()]
    nn = (1 - al - be)[:, None] * nr[:, 0] + al[:, None] * nr[:, 1] + be[:, None] * nr[:, 2]
    nn = nn / nn.norm(dim=1, keepdim=True)
    q = t[:, None] * d
    lp = light - 0.5 - q  # a light of radius 0 sits half a unit below its position on every axis
    lv = lp / lp.norm(dim=1, keepdim=True)
    dist = (light - q).norm(dim=1)
    sk, st = _hits(v32, m.vidx, torch.cat([q, lv], 1).detach(), True)
    dark = (sk >= 0) & (st < dist.detach()) & (st >= 1e-8)
    occ = albedo[order[sk.clamp(min=0)]]
    satt = torch.where(dark[:, None], occ, torch.ones_like(occ))
    col = satt * albedo[f] * (nn * lv).sum(1).clamp(min=0)[:, None]
    img = torch.full((w * h, 3), 0.9, dtype=torch.float64, device=DEV).index_put((pix,), col)
    dep = torch.zeros(w * h, dtype=torch.float64, device=DEV).index_put((pix,), t)
    gv, gl, ga = torch.autograd.grad((img, dep), (verts, light, albedo), s["grads"])
    return dict(image=img.detach(), depth=dep.detach(), vertices=gv, light=gl, albedo=ga)


def exact(case, seed):
    """Distances and gradients by brute force where that is quick; images, ids and sorted pairs are whole
    numbers, which need none."""
    k = case["kind"]
    if k == "trace" and case["rays"] * _tris(case) <= 1.2e11:
        s = prepare(case, seed)
        verts = s["mesh"].verts if case["update"] == "none" else s["verts"]
        if case["any_hit"] and case["update"] == "refit":
            return None  # the order of the first hit is that of the topology kept
        return dict(ids=None, t=_hits(verts, s["mesh"].vidx, s["rays"], case["any_hit"])[1])
    if k == "diff" and 1.4 * case["width"] * case["height"] * _tris(case) <= 1.2e11:
        s = prepare(case, seed)
        return _exact_diff(case, s)
    return None
