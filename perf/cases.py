"""The work that a program of this framework has it do, as cases that can be timed.

A case is one call (or one frame's calls) through the public Python binding over the C ABI: a rebuild, a
frame, a batch of rays, the colour stage, a path-traced image, its gradient, a batch of scenes.  Sizes are
those of the benchmark's own workloads (bench.py, rtgpu/scenes.py) and generic smaller ones.  Inputs are
made from the seed on the GPU; a handle (context, tree, captured frame) is kept by the state, as a program
keeps it from frame to frame.

Hits are rt_hit records (id and the bits of u, v, t) and trees are rt_node records, so they are returned as
whole numbers.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "raytracer-gpupro4_gb300"))
from rtgpu import autograd, scenes  # noqa: E402
from rtgpu.api import LBVH, Batch, BatchFrame, Context, Frame, Pipe, RayTracer  # noqa: E402

DEV = "cuda"
LIGHT = scenes.TORUS_LIGHT
BUILD_CLEAR_UNREACHED = 1


# ---- the cases ---------------------------------------------------------------------------------------
def listed():
    return [
        # an editor or a unit of a larger scene: the smallest rebuild, where launches are the time
        dict(name="build_1k", kind="build", scene="soup", n=1000, depth=14, flags=0),
        # one rebuild of the headline workload's mesh, as a deforming model asks for every frame
        dict(name="build_2m", kind="build", scene="ico", n=2099520, depth=20, flags=0),
        # a small interactive model, call by call: rebuild, primary rays, one shadow ray per hit
        dict(name="frame_torus_512", kind="frame", scene="torus", n=65536, depth=20, width=512, height=512, mirror=False,
             graph=False),
        # the headline workload: rebuild + primary + shadow + mirror rays at 1080p, one captured frame
        dict(name="frame_ico_1080p", kind="frame", scene="ico", n=2099520, depth=20, width=1920, height=1080,
             mirror=True, graph=True),
        # a streamed model: host vertices in, host results out, two frames in flight
        dict(name="pipe_ico_720p", kind="pipe", scene="ico", n=259920, depth=20, width=1280, height=720),
        # picking and visibility queries of a game tick: a few closest-hit rays
        dict(name="rays_pick_256", kind="rays", scene="torus", n=65536, depth=20, rays=256, any_hit=False),
        # ambient occlusion / light baking: a million incoherent any-hit rays in a random soup
        dict(name="rays_ao_1m", kind="rays", scene="soup", n=200000, depth=20, rays=1 << 20, any_hit=True),
        # the demo's own shading (colour stage with one reflection) at 720p
        dict(name="whitted_ico_720p", kind="whitted", scene="ico", n=259920, depth=20, width=1280, height=720, bounces=1),
        # an interactive path-traced preview, one sample per pixel
        dict(name="pt_preview_256", kind="pathtrace", n=16384, depth=18, width=256, height=256, spp=1, bounces=4),
        # the path-traced GI workload of the benchmark
        dict(name="pt_gi_1024", kind="pathtrace", n=262144, depth=20, width=1024, height=1024, spp=4, bounces=4),
        # the differentiable workload: image, L2 loss and gradients of one optimisation step
        dict(name="adjoint_gi_512", kind="adjoint", n=262144, depth=20, width=512, height=512, spp=8, bounces=3),
        # the batched workload: 256 uneven scenes rebuilt and traced as one captured frame
        dict(name="batch_256", kind="batch", scenes=256, lo=1000, hi=200000, sizes=4, depth=20, res=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
    """A scene kind and a triangle count that it has (any for a soup)."""
    n = _log(rng, lo, hi)
    scene = rng.choice(["soup", "torus", "ico"])
    if scene == "torus":
        minor = max(4, int(math.sqrt(n / 4)))
        n = 2 * minor * max(4, n // (2 * minor))
    elif scene == "ico":
        n = 20 * max(2, int(math.sqrt(n / 20))) ** 2
    return scene, n


def _depth(rng, n):
    """Heap depths as programs set them: enough levels for the triangles, or the configured default of 20."""
    return 20 if rng.random() < 0.7 else min(20, max(8, int(math.log2(n)) + rng.randint(1, 4)))


def draw(rng):
    kind = rng.choice(["build", "frame", "pipe", "rays", "whitted", "pathtrace", "adjoint", "batch"])
    if kind == "build":
        scene, n = _mesh(rng, 300, 2099520)
        return dict(kind=kind, scene=scene, n=n, depth=_depth(rng, n), flags=rng.choice([0, 0, BUILD_CLEAR_UNREACHED]))
    if kind == "frame":
        scene, n = _mesh(rng, 1000, 2099520)
        return dict(kind=kind, scene=scene, n=n, depth=_depth(rng, n), width=_log(rng, 97, 1920),
                    height=_log(rng, 61, 1080), mirror=rng.random() < 0.7, graph=rng.random() < 0.7)
    if kind == "pipe":
        scene, n = _mesh(rng, 1000, 500000)
        return dict(kind=kind, scene=scene, n=n, depth=_depth(rng, n), width=_log(rng, 97, 1920), height=_log(rng, 61, 1080))
    if kind == "rays":
        scene, n = _mesh(rng, 1000, 1000000)
        return dict(kind=kind, scene=scene, n=n, depth=_depth(rng, n), rays=_log(rng, 1, 3000000),
                    any_hit=rng.random() < 0.5)
    if kind == "whitted":
        scene, n = _mesh(rng, 1000, 1000000)
        return dict(kind=kind, scene=scene, n=n, depth=_depth(rng, n), width=_log(rng, 97, 1920),
                    height=_log(rng, 61, 1080), bounces=rng.randint(0, 4))
    if kind == "pathtrace":
        n = _log(rng, 1000, 262144)
        return dict(kind=kind, n=n, depth=_depth(rng, n), width=_log(rng, 61, 1024), height=_log(rng, 61, 1024),
                    spp=rng.randint(1, 4), bounces=rng.randint(0, 4))
    if kind == "adjoint":
        n = _log(rng, 1000, 262144)
        return dict(kind=kind, n=n, depth=_depth(rng, n), width=_log(rng, 61, 512), height=_log(rng, 61, 512),
                    spp=rng.randint(1, 8), bounces=rng.randint(1, 3))
    return dict(kind=kind, scenes=_log(rng, 2, 256), lo=rng.choice([300, 1000]), hi=_log(rng, 2000, 200000),
                sizes=rng.randint(0, 1 << 20), depth=rng.choice([18, 20]), res=_log(rng, 24, 256))


# ---- inputs --------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@functools.lru_cache(maxsize=4)
def _ico(n):
    s = scenes.icosphere(int(round(math.sqrt(n / 20))))
    return torch.from_numpy(s.verts).to(DEV), torch.from_numpy(s.faces).to(DEV)


def _torus_mesh(n):
    minor = max(4, int(math.sqrt(n / 4)))
    while n % (2 * minor):
        minor -= 1
    major = n // (2 * minor)
    u = torch.arange(major, device=DEV, dtype=torch.float64)[:, None] * (2 * math.pi / major)
    v = torch.arange(minor, device=DEV, dtype=torch.float64)[None, :] * (2 * math.pi / minor)
    ring = 1.0 + 0.3 * torch.cos(v)
    verts = torch.stack([ring * torch.cos(u), ring * torch.sin(u), 0.3 * torch.sin(v).expand(major, minor)], -1)
    i, j = torch.arange(major, device=DEV)[:, None], torch.arange(minor, device=DEV)[None, :]
    i1, j1 = (i + 1) % major, (j + 1) % minor
    a, b, c, d = i * minor + j, i1 * minor + j, i1 * minor + j1, i * minor + j1
    faces = torch.cat([torch.stack([a, b, c], -1).reshape(-1, 3), torch.stack([a, c, d], -1).reshape(-1, 3)])
    return verts.reshape(-1, 3), faces


def _soup(n, g):
    """Random triangles as scenes.random_soup makes them: centroids in the unit cube, edges 0.005 to 0.03."""
    c = torch.rand(n, 1, 3, device=DEV, generator=g, dtype=torch.float64)
    u = torch.randn(n, 3, 3, device=DEV, generator=g, dtype=torch.float64)
    ln = 0.005 + 0.025 * torch.rand(n, 3, 1, device=DEV, generator=g, dtype=torch.float64)
    return (c + ln * u / u.norm(dim=2, keepdim=True)).reshape(n, 9).to(torch.float32).contiguous()


def _tris(case, g):
    if case["scene"] == "soup":
        return _soup(case["n"], g)
    verts, faces = _ico(case["n"]) if case["scene"] == "ico" else _torus_mesh(case["n"])
    moved = verts + 1e-3 * torch.randn(verts.shape, device=DEV, generator=g, dtype=torch.float64)
    return moved.to(torch.float32)[faces].reshape(-1, 9).contiguous()


def _camera(case):
    if case["scene"] == "soup":
        return scenes.look_at((0.5, 0.8, -1.2), (0.5, 0.5, 0.5), width=case["width"], height=case["height"])
    return scenes.sphere_camera(case["width"], case["height"])


def _gi(case, g):
    """The GI box of scenes.gi_box with a soup of this seed: (triangles, albedo, emitter mask, radiance).  One in
    sixteen of the soup's triangles is a lamp too: in the dense soup hardly a path finds the one under the ceiling."""
    fixed = torch.from_numpy(scenes.gi_box(1).tris[:14]).to(DEV)
    tris = torch.cat([fixed, _soup(case["n"], g)]).contiguous()
    albedo = torch.cat([torch.full((12, 3), 0.75, device=DEV), torch.full((2, 3), 0.5, device=DEV),
                        0.2 + 0.6 * torch.rand(case["n"], 3, device=DEV, generator=g)]).contiguous()
    mask = torch.zeros(len(tris), device=DEV)
    mask[12:14] = 1.0
    mask[14:] = (torch.rand(case["n"], device=DEV, generator=g) < 1 / 16).float()
    return tris, albedo, mask, torch.full((3,), 10.0, device=DEV)


def _target(case, g):
    return torch.rand(case["width"] * case["height"], 3, device=DEV, generator=g)


class _DevicePtr:
    """A device array of an rt_lbvh_view as torch sees it; the tensor keeps it, and so its tree, alive."""

    def __init__(self, owner, ptr, words):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": (words,), "typestr": "<i4", "version": 3}


def _words(owner, ptr, words):
    return torch.as_tensor(_DevicePtr(owner, ptr, words), device=DEV)


def _hits(px):
    return torch.empty((px, 4), dtype=torch.int32, device=DEV)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = {"case": case, "ctx": Context(0)}
    if kind in ("pathtrace", "adjoint"):
        tris, albedo, mask, radiance = _gi(case, g)
        s["lbvh"] = LBVH(s["ctx"], len(tris), case["depth"]).Build(tris)
        s["rt"] = RayTracer(s["ctx"])
        s["cam"] = scenes.gi_camera(case["width"], case["height"])
        s["albedo"], s["mask"], s["radiance"], s["seed"] = albedo, mask, radiance, seed
        if kind == "pathtrace":
            s["emission"] = (mask[:, None] * radiance[None, :]).contiguous()
        else:
            s["albedo"].requires_grad_(True)
            s["radiance"].requires_grad_(True)
            s["target"] = _target(case, g)
        return s
    if kind == "batch":
        sizes = scenes.batch_sizes(case["scenes"], case["lo"], case["hi"], case["sizes"])
        s["tris"] = _soup(int(sizes.sum()), g)
        s["batch"] = Batch(s["ctx"], sizes, case["depth"])
        s["batch"].set_views(*scenes.batch_views(len(sizes), case["res"], case["res"]))
        s["hits"], s["vis"] = s["batch"].alloc_outputs()
        s["batch"].build(s["tris"])
        s["frame"] = BatchFrame(s["ctx"], s["batch"], s["tris"], s["hits"], s["vis"])
        return s
    s["tris"] = _tris(case, g)
    n, depth = len(s["tris"]), case["depth"]
    s["lbvh"] = LBVH(s["ctx"], n, depth)
    s["rt"] = RayTracer(s["ctx"])
    if kind == "build":
        # the tree as the next stage reads it; slots that no path reaches are never written, so they are cleared once
        s["lbvh"].Build(s["tris"], case["flags"])
        v, own = s["lbvh"].view(), s["lbvh"]
        s["tree"] = [_words(own, v.ids, n), _words(own, v.keys, n), _words(own, v.sorted_tris, 12 * n),
                     _words(own, v.nodes, 8 << depth)]
        for t in s["tree"]:
            t.zero_()
    elif kind == "rays":
        m = case["rays"]
        s["lbvh"].Build(s["tris"])
        r = torch.empty(m, 8, device=DEV)
        if case["scene"] == "soup":  # from anywhere inside, in every direction
            r[:, 0:3] = torch.rand(m, 3, device=DEV, generator=g)
        else:  # from around the object towards it
            o = torch.randn(m, 3, device=DEV, generator=g)
            r[:, 0:3] = 2.5 * o / o.norm(dim=1, keepdim=True)
        d = torch.randn(m, 3, device=DEV, generator=g)
        if case["scene"] != "soup":
            d = 0.6 * d - r[:, 0:3]
        r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
        r[:, 7] = 0.25 if case["any_hit"] and case["scene"] == "soup" else 1e16
        r.view(torch.int32)[:, 3] = -1
        s["rays"] = r
    elif kind == "whitted":
        s["lbvh"].Build(s["tris"])
        s["cam"] = _camera(case)
        m = np.zeros((6, 14), np.float32)
        rng = np.random.default_rng(seed)
        m[:, 0:3] = rng.uniform(0.0, 0.3, (6, 3))
        m[:, 3] = 1.5
        m[:, 4:7] = rng.uniform(0.2, 1.0, (6, 3))
        m[:, 7] = 0.6
        m[:, 8:11] = rng.uniform(0.0, 0.9, (6, 3))
        m[:, 11:13] = 1.0
        m[:, 13] = [1.0, 0.5, 1.0, 0.5, 1.0, 0.0]
        s["materials"] = torch.from_numpy(m).to(DEV)
        s["ids"] = torch.randint(0, 6, (n,), device=DEV, generator=g, dtype=torch.int32)
        corners = s["tris"].view(n, 3, 3)
        s["normals"] = (corners / corners.norm(dim=2, keepdim=True)).reshape(n, 9).contiguous()
    elif kind == "frame":
        px = case["width"] * case["height"]
        s["cam"], s["hits"], s["vis"] = _camera(case), _hits(px), torch.empty(px, dtype=torch.uint8, device=DEV)
        s["mirror"] = _hits(px) if case["mirror"] else None
        if case["graph"]:
            s["frame"] = Frame(s["ctx"], s["lbvh"], s["tris"], s["cam"], LIGHT, s["hits"], s["vis"], s["mirror"])
        else:
            s["leaves"] = torch.empty(px, dtype=torch.int32, device=DEV)
            s["mirror_leaves"] = torch.empty(px, dtype=torch.int32, device=DEV) if case["mirror"] else None
    else:  # pipe: pinned host vertices in, pinned host results out
        px = case["width"] * case["height"]
        s["host"] = s["tris"].cpu().pin_memory()
        s["out"] = [(torch.empty((px, 4), dtype=torch.int32).pin_memory(), torch.empty(px, dtype=torch.uint8).pin_memory(),
                     torch.empty((px, 4), dtype=torch.int32).pin_memory()) for _ in range(2)]
        s["pipe"] = Pipe(s["ctx"], s["lbvh"], n, _camera(case), LIGHT)
        s["frames"] = 0
    return s


# ---- one pass --------------------------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "build":
        s["lbvh"].Build(s["tris"], case["flags"])
        return s["tree"]
    if kind == "frame":
        if case["graph"]:
            s["frame"].launch()
        else:
            s["lbvh"].Build(s["tris"])
            s["rt"].primary_leaves(s["lbvh"], s["cam"], out=s["hits"], leaves=s["leaves"])
            s["rt"].shadow_mirror_from(s["lbvh"], s["cam"], LIGHT, s["hits"], s["leaves"], vis=s["vis"],
                                       mirror=s["mirror"], mirror_leaves=s["mirror_leaves"], with_mirror=case["mirror"])
        return [s["hits"], s["vis"], s["mirror"]]
    if kind == "pipe":
        out = s["out"][s["frames"] % 2]
        if s["frames"] >= 2:
            s["pipe"].wait(s["frames"] - 2)  # this frame's host buffers are free again
        s["pipe"].submit(s["host"], *out)
        s["frames"] += 1
        return list(out)
    if kind == "rays":
        return s["rt"].rays(s["lbvh"], s["rays"], any_hit=case["any_hit"])
    if kind == "whitted":
        return list(s["rt"].whitted(s["lbvh"], s["cam"], LIGHT, s["materials"], s["ids"], s["normals"],
                                    bounces=case["bounces"], phong=True, gloss_mapping=True, seed=7))
    if kind == "pathtrace":
        return s["rt"].pathtrace(s["lbvh"], s["albedo"], s["emission"], s["cam"], case["spp"], case["bounces"], s["seed"])
    if kind == "adjoint":
        img = autograd.render(s["albedo"], s["radiance"], s["mask"], s["rt"], s["lbvh"], s["cam"], case["spp"],
                              case["bounces"], s["seed"])
        loss = (img[:, :3] - s["target"]).square().mean()
        d_albedo, d_radiance = torch.autograd.grad(loss, [s["albedo"], s["radiance"]])
        return [img.detach(), d_albedo, d_radiance]
    s["frame"].launch()
    return [s["hits"], s["vis"]]


# ---- what a pass cannot do without -------------------------------------------------------------------------
def _walk_flops(rays, n):
    """Box tests down one root path and a leaf's triangle tests: the least a tree walk does per ray."""
    return rays * (2 * 20 * max(1.0, math.log2(max(2, n))) + 2 * 50)


def _build_bytes(n, depth):
    return 36 * n + (4 + 4 + 48) * n + 32 * min(2 * n, 1 << depth)  # soup in; ids, codes, sorted triangles, nodes out


def work(case):
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "build":
        clear = 32 * (1 << case["depth"]) if case["flags"] & BUILD_CLEAR_UNREACHED else 0
        return {"bytes": _build_bytes(n, case["depth"]) + clear, "flops": 60 * n}
    px = case.get("width", 0) * case.get("height", 0)
    if kind in ("frame", "pipe"):
        both = kind == "pipe" or case["mirror"]
        out = px * (16 + 1 + (16 if both else 0))
        return {"bytes": _build_bytes(n, case["depth"]) + out, "flops": 60 * n + _walk_flops(px, n)}
    if kind == "rays":
        return {"bytes": case["rays"] * (32 + 16) + 48 * min(n, case["rays"]), "flops": _walk_flops(case["rays"], n)}
    if kind == "whitted":
        return {"bytes": 32 * px + (48 + 36 + 4) * min(n, px), "flops": _walk_flops(px * (case["bounces"] + 1), n)}
    if kind in ("pathtrace", "adjoint"):
        paths = px * case["spp"] * (case["bounces"] + 1)
        both = 1 if kind == "pathtrace" else 2
        return {"bytes": both * (16 * px + (48 + 24) * n) + (12 * n + 12 * px if both == 2 else 0),
                "flops": both * _walk_flops(paths, n)}
    sizes = scenes.batch_sizes(case["scenes"], case["lo"], case["hi"], case["sizes"])
    px = case["scenes"] * case["res"] ** 2
    return {"bytes": sum(_build_bytes(int(k), case["depth"]) for k in sizes) + 17 * px,
            "flops": 60 * int(sizes.sum()) + sum(_walk_flops(case["res"] ** 2, int(k)) for k in sizes)}


# ---- the path-traced image and its gradient in 64 bits ---------------------------------------------------------
_M64 = (1 << 64) - 1


def _i64(v):
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _shr(x, k):
    """Logical right shift of int64 by a constant."""
    return (x >> k) & ((1 << (64 - k)) - 1)


class _Pcg:
    """One PCG32 stream per path (O'Neill 2014), seeded by splitmix64 of (seed, pixel, sample)."""

    def __init__(self, seed, pixel, sample):
        z = (pixel * 65536 + sample + 1) * _i64(0x9E3779B97F4A7C15) + _i64(seed) + _i64(0x9E3779B97F4A7C15)
        z = (z ^ _shr(z, 30)) * _i64(0xBF58476D1CE4E5B9)
        z = (z ^ _shr(z, 27)) * _i64(0x94D049BB133111EB)
        z = z ^ _shr(z, 31)
        self.inc = (pixel << 1) | 1
        self.state = torch.zeros_like(pixel)
        on = torch.ones_like(pixel, dtype=torch.bool)
        self.next(on)
        self.state = self.state + z
        self.next(on)

    def next(self, on):
        old = self.state
        self.state = torch.where(on, old * 6364136223846793005 + self.inc, old)
        x = _shr(_shr(old, 18) ^ old, 27) & 0xFFFFFFFF
        rot = _shr(old, 59)
        return ((x >> rot) | (x << (32 - rot))) & 0xFFFFFFFF

    def uniform(self, on):
        return (self.next(on) >> 8).double() / 16777216.0


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _closest(tris, o, d, exclude, pairs=1 << 25):
    """Closest triangle of each ray by testing all of them: (id or -1, t)."""
    A, B, C = tris[:, 0:3], tris[:, 3:6], tris[:, 6:9]
    e1, e2 = B - A, C - A
    nrm = torch.linalg.cross(e1, e2)
    # t = ((A - o) . n) / (d . n); with w = d x (A - o): u = -(e2 . w) / (d . n), v = (e1 . w) / (d . n)
    c_a, c_1, c_2 = _dot(A, nrm)[:, 0], torch.linalg.cross(e1, A), torch.linalg.cross(e2, A)
    ids, ts = [], []
    step = max(1, pairs // len(tris))
    for k in range(0, len(o), step):
        p, q = o[k:k + step], d[k:k + step]
        m = torch.linalg.cross(q, p)
        dn = q @ nrm.T
        t = (c_a[None] - p @ nrm.T) / dn
        # e . (d x (A - o)) = -(d . (e x A)) - e . (d x o)
        w2 = -(q @ c_2.T) - m @ e2.T
        w1 = -(q @ c_1.T) - m @ e1.T
        u, v = -w2 / dn, w1 / dn
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= 0)
        t = torch.where(ok, t, torch.inf)
        x = exclude[k:k + step]
        has = x >= 0
        t[torch.nonzero(has)[:, 0], x[has]] = torch.inf
        best, at = t.min(dim=1)
        ids.append(torch.where(torch.isfinite(best), at, -1))
        ts.append(best)
    return torch.cat(ids), torch.cat(ts)


def _exact_image(case, seed, tris, albedo, emission):
    """The mean over samples of the paths' radiance, differentiable in albedo and emission."""
    w, h, spp, bounces = case["width"], case["height"], case["spp"], case["bounces"]
    cam = scenes.gi_camera(w, h)
    vec = lambda a: torch.tensor(list(a), device=DEV, dtype=torch.float64)  # noqa: E731
    px = torch.arange(w * h, device=DEV)
    i, j = (px % w).double(), (px // w).double()
    image = 0.0
    for n in range(spp):
        g = _Pcg(seed, px, n)
        on = torch.ones_like(px, dtype=torch.bool)
        jx, jy = 2 * g.uniform(on) - 1, 2 * g.uniform(on) - 1
        x, y = (2 * i + 1 - w + jx) / h, -(2 * j + 1 - h + jy) / h
        d = vec(cam.right) * (x * cam.tan_half_fovy)[:, None] + vec(cam.up) * (y * cam.tan_half_fovy)[:, None] + vec(cam.fwd)
        d = d / d.norm(dim=1, keepdim=True)
        o = vec(cam.eye).expand_as(d)
        live, last = on, torch.full_like(px, -1)
        beta, radiance = torch.ones_like(d), torch.zeros_like(d)
        for s in range(bounces + 1):
            hit, t = _closest(tris, o, d, last)
            at = hit.clamp(min=0)
            miss = live & (hit < 0)
            radiance = radiance + torch.where(miss[:, None], beta, 0.0)  # a white sky
            live = live & (hit >= 0)
            radiance = radiance + torch.where(live[:, None], beta * emission[at], 0.0)
            beta = torch.where(live[:, None], beta * albedo[at], beta)
            if s == bounces:
                break
            tri = tris[at]
            nrm = torch.linalg.cross(tri[:, 3:6] - tri[:, 0:3], tri[:, 6:9] - tri[:, 0:3])
            nrm = nrm / nrm.norm(dim=1, keepdim=True)
            nrm = torch.where(_dot(nrm, d) > 0, -nrm, nrm)
            # a point on the disc by rejection, lifted to the hemisphere (Malley); basis of Duff et al. 2017
            a, b, need = torch.zeros_like(x), torch.zeros_like(x), live.clone()
            while bool(need.any()):
                p, q = 2 * g.uniform(need) - 1, 2 * g.uniform(need) - 1
                a, b = torch.where(need, p, a), torch.where(need, q, b)
                need = need & (a * a + b * b > 1)
            z = (1 - a * a - b * b).clamp(min=0).sqrt()
            nx, ny, nz = nrm.unbind(1)
            sign = torch.copysign(torch.ones_like(nz), nz)
            k = -1 / (sign + nz)
            m = nx * ny * k
            T = torch.stack([1 + sign * nx * nx * k, sign * m, -sign * nx], 1)
            B = torch.stack([m, sign + ny * ny * k, -ny], 1)
            o = torch.where(live[:, None], o + torch.where(live, t, 0.0)[:, None] * d, o)
            d = torch.where(live[:, None], T * a[:, None] + B * b[:, None] + nrm * z[:, None], d)
            last = torch.where(live, hit, last)
        image = image + radiance / spp
    return torch.cat([image, torch.ones_like(image[:, :1])], 1)


def exact(case, seed):
    """The images and gradients of the path tracer by brute force, where that ends within seconds.  Hits,
    visibilities and trees are whole numbers; the colour stage's images take too long at every size above a
    toy's, and no size of its range is one."""
    if case["kind"] not in ("pathtrace", "adjoint"):
        return None
    pairs = case["n"] * case["width"] * case["height"] * case["spp"] * (case["bounces"] + 1)
    if pairs > 1.2e10:
        return None
    g = _gen(seed)
    tris, albedo, mask, radiance = _gi(case, g)
    tris, albedo, mask, radiance = tris.double(), albedo.double(), mask.double(), radiance.double()
    if case["kind"] == "pathtrace":
        return _exact_image(case, seed, tris, albedo, mask[:, None] * radiance[None, :])
    target = _target(case, g).double()
    albedo.requires_grad_(True)
    radiance.requires_grad_(True)
    img = _exact_image(case, seed, tris, albedo, mask[:, None] * radiance[None, :])
    loss = (img[:, :3] - target).square().mean()
    d_albedo, d_radiance = torch.autograd.grad(loss, [albedo, radiance])
    return [img.detach(), d_albedo, d_radiance]
