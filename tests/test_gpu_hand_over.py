"""Closest hits do not depend on who traces the ray: its lane, a warp of its own (calls of
few rays, rays over the hand-over budget) or one lane of that warp.  Where surfaces coincide, the hit
depends on the order in which leaves are entered, to the last bit of a distance, so the
scenes here overlap: triangles in one plane (leaves whose entry distance lies above a hit's
by a rounding), rays along the faces of boxes (NaN distances), and layers that come nearer
and nearer in the order of the walk (more pending hits than are kept).  Hits are the oracle's
on their bits, for every budget and number of rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUDGETS = (None, 0, 1, 40)


def coplanar(n, seed, tilt=False):
    rng = np.random.default_rng(seed)
    v = rng.uniform(0, 1, (n, 1, 2)) + rng.uniform(-0.2, 0.2, (n, 3, 2))
    p = np.concatenate([v, np.full((n, 3, 1), 0.3)], 2)
    if tilt:
        p = p @ np.linalg.qr(rng.normal(size=(3, 3)))[0]
    return np.ascontiguousarray(p.reshape(n, 9), np.float32)


def ground(k, seed):
    """A k x k grid of squares at exact coordinates in the plane z = 0.3 and, in the same
    plane, larger triangles with corners on the grid."""
    i, j = np.meshgrid(np.arange(k), np.arange(k), indexing="ij")
    a = np.stack([i, j], -1).reshape(-1, 2) / 16.0
    s = np.array([[0, 0], [1, 0], [1, 1], [0, 0], [1, 1], [0, 1]]) / 16.0
    sq = (a[:, None] + s[None]).reshape(-1, 3, 2)
    rng = np.random.default_rng(seed)
    big = rng.integers(0, k + 1, (k * k, 3, 2)) / 16.0
    p = np.concatenate([sq, big])
    p = np.concatenate([p, np.full(p.shape[:2] + (1,), 0.3)], 2)
    return np.ascontiguousarray(p.reshape(-1, 9), np.float32)


def layers(n):
    """Sheets whose centroids move along +x and which a ray along +x meets at falling x."""
    c = np.linspace(0.0, 1.0, n)
    slope = 2.0 - 2.0 * c
    y = np.array([-4.0, 0.5, 0.5])
    z = np.array([0.0, -3.0, 3.0])
    x = c[:, None] + slope[:, None] * (y[None] + 1.0)
    return np.stack([x, np.broadcast_to(y, x.shape), np.broadcast_to(z, x.shape)], -1).reshape(n, 9).astype(np.float32)


def rays_at(tris, n, seed):
    rng = np.random.default_rng(seed)
    t = tris[rng.integers(0, len(tris), n)].reshape(n, 3, 3).mean(1)
    o = t + rng.normal(size=(n, 3))
    d = t - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return o.astype(np.float32), d.astype(np.float32)


def down_at(k, n, seed):
    """Straight down through grid points and along grid lines."""
    rng = np.random.default_rng(seed)
    xy = rng.integers(0, 2 * k + 1, (n, 2)) / 32.0
    free = rng.random(n) < 0.3
    xy[free, 1] = rng.uniform(0, k / 16.0, free.sum())
    o = np.concatenate([xy, np.full((n, 1), 2.0)], 1)
    d = np.broadcast_to(np.array([0.0, 0.0, -1.0]), (n, 3))
    return o.astype(np.float32), np.ascontiguousarray(d, np.float32)


def case(kind, n):
    if kind == "plane":
        tris = coplanar(3000, 5)
        return tris, 16, rays_at(tris, n, n)
    if kind == "few leaves":
        tris = coplanar(300, 5)
        return tris, 16, rays_at(tris, n, n)
    if kind == "tilted":
        tris = coplanar(2000, 6, True)
        return tris, 16, rays_at(tris, n, n)
    if kind == "down":
        return ground(40, 3), 20, down_at(40, n, n)
    tris = layers(500)
    rng = np.random.default_rng(n)
    o = np.stack([np.full(n, -1.0), rng.uniform(-0.01, 0.01, n), rng.uniform(-0.01, 0.01, n)], 1)
    d = np.stack([np.ones(n), rng.uniform(-1e-3, 1e-3, n), rng.uniform(-1e-3, 1e-3, n)], 1)
    return tris, 20, (o.astype(np.float32), d.astype(np.float32))


@pytest.mark.parametrize("n", [31, 16384, 16385, 30000])
@pytest.mark.parametrize("kind", ["plane", "few leaves", "tilted", "down", "layers"])
def test_rays(gpu_ctx, oracle_mod, kind, n):
    import torch
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris, depth, (o, d) = case(kind, n)
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    tmax, excl = np.full(n, 1e16, np.float32), np.full(n, -1, np.int32)
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax, excl))
    excl2 = np.where(np.arange(n) % 2 == 0, ref["id"], -1).astype(np.int32)
    tmax2 = np.where(np.arange(n) % 5 == 0, ref["t"], 1e16).astype(np.float32)  # a bound at a hit's distance
    ref2 = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax2, excl2))
    rt = RayTracer(gpu_ctx)
    same = lambda a, b: np.array_equal(hits_to_numpy(a).view(np.int32), b.view(np.int32))  # noqa: E731
    try:
        for budget in BUDGETS:
            gpu_ctx.set_trace_budget(budget)
            assert same(rt.rays(lb, rays_tensor(o, d, tmax, excl, "cuda")), ref), budget
            assert same(rt.rays(lb, rays_tensor(o, d, tmax2, excl2, "cuda")), ref2), budget
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)
    assert (ref["id"] >= 0).mean() > 0.2


@pytest.mark.parametrize("kind", ["plane", "tilted", "down"])
def test_restarted_rays(gpu_ctx, oracle_mod, kind):
    """The order of a restarted walk begins at its start node."""
    import ctypes as C

    import torch
    from rtgpu import _lib as L
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    n = 20000
    tris, depth, (o, d) = case(kind, n)
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, reached = oracle_mod.lbvh_build(tris, depth)
    leaf = np.nonzero((reached != 0) & ((nodes["prim_count"] & 4) != 0))[0]
    starts = leaf[np.random.default_rng(1).integers(0, len(leaf), n)].astype(np.uint32)
    tmax, excl = np.full(n, 1e16, np.float32), np.full(n, -1, np.int32)
    ref, ref_leaves = oracle_mod.trace_from(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax, excl), starts)
    st = torch.from_numpy(starts.view(np.int32)).cuda()
    rt = RayTracer(gpu_ctx)
    try:
        for budget in BUDGETS:
            gpu_ctx.set_trace_budget(budget)
            got, leaves = rt.rays_from(lb, rays_tensor(o, d, tmax, excl, "cuda"), st)
            assert np.array_equal(hits_to_numpy(got).view(np.int32), ref.view(np.int32)), budget
            assert np.array_equal(leaves.cpu().numpy().view(np.uint32), ref_leaves), budget
            for m in (9000, n):  # a warp a ray or a lane, without leaves
                hits = torch.empty((m, 4), dtype=torch.int32, device="cuda")
                ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
                dev = rays_tensor(o[:m], d[:m], tmax[:m], excl[:m], "cuda")
                assert L.lib().rt_trace_rays_from(gpu_ctx.h, lb.h, ptr(dev), m, 0, ptr(st), ptr(hits), None, None) == L.RT_OK
                assert np.array_equal(hits_to_numpy(hits).view(np.int32), ref[:m].view(np.int32)), (budget, m)
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)


@pytest.mark.parametrize("block", [0, 2, 7])
@pytest.mark.parametrize("kind", ["plane", "tilted"])
def test_frame(gpu_ctx, oracle_mod, kind, block):
    """Primary, shadow and mirror rays and their leaves under every budget."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy
    tris, depth, _ = case(kind, 1)
    flat = tris.reshape(-1, 3)
    c = flat.mean(0)
    eye = c + np.array([0.1, 0.4, 1.3]) * (1 if kind == "plane" else -1)
    cam = scenes.look_at(eye, c, width=321, height=201)
    light = tuple(float(x) for x in eye + np.array([0.7, 0.2, 0.1]))
    walls = np.concatenate([tris, tris[:600] + np.float32(0.02)])  # something to mirror and to cast shadows
    lb = LBVH(gpu_ctx, len(walls), depth).Build(torch.from_numpy(walls).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(walls, depth)
    ref, ref_leaves = oracle_mod.trace_from(nodes, depth, ids, walls, oracle_mod.primary_rays(cam))
    ref_vis, ref_mir, ref_ml = oracle_mod.shadow_mirror_from(nodes, depth, ids, walls, cam, light, ref, ref_leaves)
    rt = RayTracer(gpu_ctx)
    gpu_ctx.set_heavy_block(block)
    try:
        for budget in (0, None, 1, 40):
            gpu_ctx.set_trace_budget(budget)
            prim, leaves = rt.primary_leaves(lb, cam)
            assert np.array_equal(hits_to_numpy(prim).view(np.int32), ref.view(np.int32)), budget
            assert np.array_equal(leaves.cpu().numpy().view(np.uint32), ref_leaves), budget
            vis, mir, ml = rt.shadow_mirror_from(lb, cam, light, prim, leaves)
            assert np.array_equal(vis.cpu().numpy(), ref_vis), budget
            assert np.array_equal(hits_to_numpy(mir).view(np.int32), ref_mir.view(np.int32)), budget
            assert np.array_equal(ml.cpu().numpy().view(np.uint32), ref_ml), budget
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)
        gpu_ctx.set_heavy_block(None)
    assert (ref["id"] >= 0).mean() > 0.2 and len(np.unique(ref_vis)) >= 3 and (ref_mir["id"] >= 0).any()


@pytest.mark.parametrize("n", [9000, 60000])
@pytest.mark.parametrize("scale,offset,stretch", [(1e-18, 1e5, (1, 1, 1)), (1e4, 1e7, (1, 1e-7, 1e3)), (1e4, 1e5, (1, 1e-3, 1)),
                                                  (1.0, 0.0, (1, 1, 0))])
def test_rays_along_faces(gpu_ctx, oracle_mod, scale, offset, stretch, n):
    """Far from the origin of coordinates few values are left between the triangles, and rays in a
    plane x = const run along the faces of many boxes."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris = scenes.random_soup(6000, 7, 0.01, 0.1).reshape(-1, 3) * np.array(stretch) + offset
    tris = tris * scale
    tris = np.ascontiguousarray(tris.reshape(-1, 9), np.float32)
    rng = np.random.default_rng(n)
    size = float((tris.reshape(-1, 3).max(0) - tris.reshape(-1, 3).min(0)).max())
    t = tris[rng.integers(0, len(tris), n)].reshape(n, 3, 3).mean(1).astype(np.float64)
    d = rng.normal(size=(n, 3))
    d[:, 0] = 0.0
    d[::5, 1] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (t - d * size * rng.choice([0.0, 0.01, 0.5, 14.0, 1e3], n)[:, None]).astype(np.float32)
    d = d.astype(np.float32)
    lb = LBVH(gpu_ctx, len(tris), 16).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, 16)
    tmax, excl = np.full(n, 1e16, np.float32), np.full(n, -1, np.int32)
    rays = oracle_mod.rays_array(o, d, tmax, excl)
    ref = oracle_mod.trace(nodes, 16, ids, tris, rays)
    any_ref = oracle_mod.trace(nodes, 16, ids, tris, rays, any_hit=True)
    rt, dev = RayTracer(gpu_ctx), rays_tensor(o, d, tmax, excl, "cuda")
    try:
        for budget in BUDGETS:
            gpu_ctx.set_trace_budget(budget)
            assert np.array_equal(hits_to_numpy(rt.rays(lb, dev)).view(np.int32), ref.view(np.int32)), budget
            assert np.array_equal(hits_to_numpy(rt.rays(lb, dev, any_hit=True))["id"] >= 0, any_ref["id"] >= 0), budget
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)
    assert (ref["id"] >= 0).mean() > 0.2
