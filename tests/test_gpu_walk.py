"""The walk over the trace records (Walk in rt_traverse.cuh) where it can go
wrong, against the oracle: leaves around the sizes that change their form
(a word holds fewer than 32 triangles, larger leaves are box-tested first; more
than 2 or 3 are pooled), trees of one leaf and of flat scenes, rays that the
records do not serve (a zero direction component, an origin far outside, very
short and very long directions), ray counts around a warp and around the
number up to which a ray gets a warp, and any-hit rays around the hand-over
budget.  Hits are compared on their bits: the walk accepts a triangle under
the reference's own tests, so no tolerance is needed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(kind):
    from rtgpu import scenes
    if kind == "one":
        return scenes.random_soup(1, 5), 8
    if kind == "one_leaf":  # equal codes: a root leaf of 40 triangles
        return np.repeat(scenes.random_soup(1, 6), 40, 0) + np.linspace(0, 1e-6, 40, dtype=np.float32)[:, None], 8
    if kind == "leaf_sizes":  # clusters of 1 .. 36 near-equal triangles and one of 300
        base = scenes.random_soup(37, 7, 0.02, 0.1)
        sizes = list(range(1, 37)) + [300]
        tris = np.concatenate([np.repeat(base[i:i + 1], m, 0) for i, m in enumerate(sizes)])
        return tris + np.random.default_rng(1).normal(0, 1e-6, tris.shape).astype(np.float32), 12
    if kind == "flat":  # no extent in z
        tris = scenes.random_soup(3000, 8, 0.01, 0.05)
        tris.reshape(-1, 3, 3)[..., 2] = 0.25
        return tris, 14
    if kind == "offset":  # far from the origin of coordinates
        return scenes.random_soup(3000, 9, 0.02, 0.1) + np.float32(300.0), 14
    return scenes.random_soup(20000, 10), 16


def rays_for(tris, n, seed):
    rng = np.random.default_rng(seed)
    lo, hi = tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)
    size = max(float((hi - lo).max()), 1e-3)
    o = rng.uniform(lo - 0.5 * size, hi + 0.5 * size, (n, 3))
    target = tris[rng.integers(0, len(tris), n)].reshape(n, 3, 3).mean(1)
    d = target - o + rng.normal(0, 0.02 * size, (n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    k = np.arange(n)
    far = k % 7 == 1           # out of the records' range
    o[far] -= 40.0 * size * d[far]
    axis = k % 7 == 2          # along an axis: two infinite 1 / d
    d[axis] = np.eye(3)[k[axis] % 3] * np.where(k[axis] % 2, 1.0, -1.0)[:, None]
    o[axis] = target[axis] - size * d[axis]
    plane = k % 7 == 3         # one infinite 1 / d
    d[plane, 2] = 0.0
    d[k % 14 == 4] *= 1e-4
    d[k % 14 == 11] *= 1e5
    tmax = np.where(k % 5 == 0, 0.7 * size, 1e16)
    excl = np.where(k % 3 == 0, rng.integers(0, len(tris), n), -1)
    return o.astype(np.float32), d.astype(np.float32), tmax.astype(np.float32), excl.astype(np.int32)


@pytest.mark.parametrize("kind,n", [("one", 1), ("one_leaf", 33), ("leaf_sizes", 4000), ("leaf_sizes", 16385), ("flat", 17000),
                                    ("offset", 17000), ("soup", 31), ("soup", 16384), ("soup", 16385), ("soup", 40000)])
def test_closest_hits(gpu_ctx, oracle_mod, kind, n):
    import torch
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris, depth = scene(kind)
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    o, d, tmax, excl = rays_for(tris, n, 3)
    rays = rays_tensor(o, d, tmax, excl, "cuda")
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax, excl))
    rt = RayTracer(gpu_ctx)
    got = hits_to_numpy(rt.rays(lb, rays))
    gpu_ctx.check()
    assert np.array_equal(got.view(np.int32), ref.view(np.int32))
    # with leaves (always the walk), from the root and restarted at the hits' leaves
    hits, leaves = rt.rays_from(lb, rays, None)
    again, leaves2 = rt.rays_from(lb, rays, leaves)
    gpu_ctx.check()
    assert np.array_equal(hits_to_numpy(hits).view(np.int32), ref.view(np.int32))
    assert np.array_equal(hits_to_numpy(again).view(np.int32), ref.view(np.int32))
    assert torch.equal(leaves, leaves2)
    if n > 30:
        assert (ref["id"] >= 0).mean() > 0.2


@pytest.mark.parametrize("budget,n", [(0, 9001), (60, 9001), (0, 1 << 20), (24, (1 << 20) + 1), (384, (1 << 20) + 33)])
def test_any_hit_budget(gpu_ctx, oracle_mod, budget, n):
    """The first hit of a ray that stays within the budget is traverse()'s; one
    that does not still reports a hit exactly when there is one."""
    import torch
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris, depth = scene("soup")
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    o, d, tmax, excl = rays_for(tris, n, 4)
    ref, st = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax, excl), any_hit=True, stats=True)
    gpu_ctx.set_trace_budget(budget)
    try:
        got = hits_to_numpy(RayTracer(gpu_ctx).rays(lb, rays_tensor(o, d, tmax, excl, "cuda"), any_hit=True))
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)
    assert np.array_equal(got["id"] >= 0, ref["id"] >= 0)
    within = (st.sum(1) <= budget) if budget else np.ones(len(ref), bool)
    assert np.array_equal(got[within].view(np.int32), ref[within].view(np.int32))
    assert within.sum() > 100 and (budget == 0 or (~within).sum() > 100)


@pytest.mark.parametrize("w,h,spp,bounces", [(1, 1, 2, 0), (33, 17, 3, 3), (64, 48, 5, 2)])
def test_samples_traced_apart(gpu_ctx, oracle_mod, w, h, spp, bounces):
    """Several samples a pixel are paths of their own whose terms are folded in
    order: the image of spp calls of one sample each, bit for bit."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer
    gi = scenes.gi_box(500, seed=11)
    lb = LBVH(gpu_ctx, len(gi.tris), 14).Build(torch.from_numpy(gi.tris).cuda())
    alb, em = torch.from_numpy(gi.albedo).cuda(), torch.from_numpy(gi.emission).cuda()
    cam = scenes.gi_camera(w, h)
    rt = RayTracer(gpu_ctx)
    img = rt.pathtrace(lb, alb, em, cam, spp, bounces, 9)
    one = rt.pathtrace(lb, alb, em, cam, 1, bounces, 9)
    for k in range(1, spp):
        one = rt.pathtrace(lb, alb, em, cam, 1, bounces, 9, out=one, first_sample=k)
    gpu_ctx.check()
    assert torch.equal(img.view(torch.int32), one.view(torch.int32))
    nodes, ids, _, _ = oracle_mod.lbvh_build(gi.tris, 14)
    ref = oracle_mod.pathtrace(nodes, 14, ids, gi.tris, gi.albedo, gi.emission, cam, spp, bounces, 9)
    assert np.array_equal(img.cpu().numpy().view(np.int32).ravel(), np.ascontiguousarray(ref, np.float32).view(np.int32).ravel())


@pytest.mark.parametrize("first,then", [("build", "build"), ("import", "build"), ("build", "import")])
def test_captured_trace_over_a_later_tree(gpu_ctx, oracle_mod, first, then):
    """A captured trace call makes the records of the tree that is there when it
    is replayed, whoever made that tree."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import Context, LBVH, RayTracer, hits_to_numpy
    n, depth = 20000, 16
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=150, height=90)
    soups = [scenes.random_soup(n, 21), scenes.random_soup(n - 700, 22)]
    dev = [torch.from_numpy(s).cuda() for s in soups]
    stream = torch.cuda.Stream()
    ctx = Context(0, stream)
    lb, rt = LBVH(ctx, n, depth), RayTracer(ctx)

    def put(how, i):
        if how == "build":
            lb.Build(dev[i])
        else:
            nodes, ids, _, _ = oracle_mod.lbvh_build(soups[i], depth)
            lb.Import(nodes, ids, soups[i])

    torch.cuda.synchronize()
    out = torch.empty((cam.width * cam.height, 4), dtype=torch.int32, device="cuda")
    put(first, 0)
    rt.primary(lb, cam, out=out)
    stream.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        rt.primary(lb, cam, out=out)
    put(then, 1)
    stream.synchronize()
    g.replay()
    torch.cuda.synchronize()
    ctx.check()
    nodes, ids, _, _ = oracle_mod.lbvh_build(soups[1], depth)
    ref = oracle_mod.trace(nodes, depth, ids, soups[1], oracle_mod.primary_rays(cam))
    assert np.array_equal(hits_to_numpy(out).view(np.int32).ravel(), np.ascontiguousarray(ref).view(np.int32).ravel())
    assert (ref["id"] >= 0).mean() > 0.2


def test_images_of_many_tiles(gpu_ctx, oracle_mod):
    """The variants for more than eight tiles a warp: an image against the oracle, a
    batch against two halves of it that take the other variant."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import Batch, LBVH, RayTracer, hits_to_numpy
    tris, depth = scene("soup")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tiles = 8 * 32 * sms + 1
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=1600, height=4 * -(-tiles // 200))
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    got = hits_to_numpy(RayTracer(gpu_ctx).primary(lb, cam))
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.primary_rays(cam))
    gpu_ctx.check()
    assert np.array_equal(got.view(np.int32), ref.view(np.int32))

    counts = scenes.batch_sizes(2 * (-(-tiles // 1024)), 300, 3000, 5)  # 1,024 tiles a scene
    soup = torch.from_numpy(scenes.random_soup(int(counts.sum()), 6, 0.02, 0.1)).cuda()
    cams, lights = scenes.batch_views(len(counts), 256, 128)
    half = len(counts) // 2
    cut = int(counts[:half].sum())

    def traced(c, t, k, li, shadow):
        b = Batch(gpu_ctx, c, 14)
        b.set_views(k, li)
        hits, vis = b.alloc_outputs(shadow)
        b.build(t.contiguous())
        b.trace(hits, vis)
        gpu_ctx.check()
        return hits.reshape(-1), vis

    for shadow in (True, False):
        whole, vis = traced(counts, soup, cams, lights, shadow)
        parts = [traced(counts[:half], soup[:cut], cams[:half], lights[:half], shadow),
                 traced(counts[half:], soup[cut:], cams[half:], lights[half:], shadow)]
        assert torch.equal(whole.view(torch.int32), torch.cat([p[0] for p in parts]).view(torch.int32))
        if shadow:
            assert torch.equal(vis.reshape(-1), torch.cat([p[1].reshape(-1) for p in parts]))


@pytest.mark.parametrize("budget", [0, 1, 200, None])
def test_colour_stage_hands_over_shadow_rays(gpu_ctx, oracle_mod, budget):
    """Shadow rays traced by their lane, by a warp, or handed over once the list is
    empty: the oracle's image."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer
    from test_gpu_whitted import materials
    tris, depth = scene("soup")
    mats = materials()
    mids = np.random.default_rng(2).integers(0, len(mats), len(tris)).astype(np.int32)
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=183, height=97)
    light = (0.5, 3.0, 0.4)
    gpu_ctx.set_trace_budget(budget)
    try:
        acc, _ = RayTracer(gpu_ctx).whitted(lb, cam, light, mats, torch.from_numpy(mids).cuda(), bounces=2, shadows=True)
        gpu_ctx.check()
    finally:
        gpu_ctx.set_trace_budget(None)
    ref, _ = oracle_mod.render_whitted(nodes, depth, ids, tris, cam, light, mats, mids, None, bounces=2, shadows=True)
    got = acc.cpu().numpy()
    assert np.array_equal(got.view(np.int32).ravel(), np.ascontiguousarray(ref, np.float32).view(np.int32).ravel())
    assert ref[:, :3].max() > 0.1
