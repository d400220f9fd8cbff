"""Calls under the context's limits (rt_ctx_set_limit): the radiance terms of a call of several
samples in chunks and without scratch, in and beside a stream capture; the adjoint in several launches;
more rays over the budget than their list holds; trees and batches without trace records.  Each does
the work that it does without the limit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def limit(gpu_ctx):
    from rtgpu import _lib as L
    yield lambda which, value: gpu_ctx.set_limit(getattr(L, "RT_LIMIT_" + which), value)
    for k in range(4):
        gpu_ctx.set_limit(k, None)
    gpu_ctx.set_trace_budget(None)


def gi(ctx, n=500, depth=14):
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH
    g = scenes.gi_box(n, seed=11)
    lb = LBVH(ctx, len(g.tris), depth).Build(torch.from_numpy(g.tris).cuda())
    return g, lb, torch.from_numpy(g.albedo).cuda(), torch.from_numpy(g.emission).cuda()


def same(a, b):
    import torch
    return torch.equal(a.view(torch.int32), b.view(torch.int32))


def test_refused(gpu_ctx):
    from rtgpu import _lib as L
    lib = L.lib()
    for which, value in ((L.RT_LIMIT_PATHS, 31), (L.RT_LIMIT_PATHS, (1 << 31) + 1), (L.RT_LIMIT_RECHECKED_RAYS, 0),
                         (L.RT_LIMIT_RECHECKED_RAYS, (1 << 20) + 1), (4, 1)):
        assert lib.rt_ctx_set_limit(gpu_ctx.h, which, value) == L.RT_ERR_INVALID
    assert lib.rt_ctx_set_limit(None, 0, 0) == L.RT_ERR_INVALID


@pytest.mark.parametrize("w,h,spp,held", [(33, 17, 5, 2), (33, 17, 6, 3), (64, 48, 4, 3), (1, 70, 3, 2)])
def test_path_scratch(gpu_ctx, oracle_mod, limit, w, h, spp, held):
    """Scratch for `held` samples at a time (the last chunk may be shorter), for one, and none; a call
    that continues an image."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import RayTracer
    g, lb, alb, em = gi(gpu_ctx)
    cam, rt, bounces = scenes.gi_camera(w, h), RayTracer(gpu_ctx), 3
    nodes, ids, _, _ = oracle_mod.lbvh_build(g.tris, 14)
    ref = oracle_mod.pathtrace(nodes, 14, ids, g.tris, g.albedo, g.emission, cam, spp + 2, bounces, 9)
    sample = w * h * ((bounces + 1) * 12 + 1)
    for nbytes in (held * sample, (held + 1) * sample - 1, sample, 0, None):
        limit("PATH_SCRATCH", nbytes)
        img = rt.pathtrace(lb, alb, em, cam, 2, bounces, 9)
        img = rt.pathtrace(lb, alb, em, cam, spp, bounces, 9, out=img, first_sample=2)
        gpu_ctx.check()
        assert np.array_equal(img.cpu().numpy().view(np.int32).ravel(), np.ascontiguousarray(ref, np.float32).view(np.int32).ravel())


def test_path_scratch_is_given_back(gpu_ctx, limit):
    import torch
    from rtgpu import scenes
    from rtgpu.api import RayTracer
    g, lb, alb, em = gi(gpu_ctx)
    rt, cam = RayTracer(gpu_ctx), scenes.gi_camera(1024, 1024)
    limit("PATH_SCRATCH", 0)
    img = rt.pathtrace(lb, alb, em, cam, 8, 3, 9)
    gpu_ctx.sync()
    free = torch.cuda.mem_get_info()[0]
    rt.pathtrace(lb, alb, em, cam, 8, 3, 9, out=img)
    gpu_ctx.sync()
    assert torch.cuda.mem_get_info()[0] == free  # a call without scratch allocates nothing
    limit("PATH_SCRATCH", None)
    rt.pathtrace(lb, alb, em, cam, 8, 3, 9, out=img)
    gpu_ctx.sync()
    assert torch.cuda.mem_get_info()[0] <= free - (300 << 20)
    limit("PATH_SCRATCH", 100 << 20)
    assert torch.cuda.mem_get_info()[0] == free


def test_captured_samples(oracle_mod, rt_lib):
    """A call of several samples in a stream capture, and one that must allocate while another
    thread captures in the global mode."""
    import threading
    import torch
    from rtgpu import scenes
    from rtgpu.api import Context, RayTracer
    stream, other = torch.cuda.Stream(), torch.cuda.Stream()
    ctx, ctx2 = Context(0, stream), Context(0, other)
    g, lb, alb, em = gi(ctx)
    torch.cuda.synchronize()
    cam, rt = scenes.gi_camera(65, 33), RayTracer(ctx)
    ref = rt.pathtrace(lb, alb, em, cam, 3, 2, 9)
    img = torch.zeros_like(ref)
    img2 = torch.zeros_like(ref)
    torch.cuda.synchronize()
    out = {}

    def beside():
        try:
            RayTracer(ctx2).pathtrace(lb, alb, em, cam, 3, 2, 9, out=img2)  # allocates its scratch
        except Exception as e:  # noqa: BLE001
            out["error"] = e

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="global"):
        rt.pathtrace(lb, alb, em, cam, 3, 2, 9, out=img)
        t = threading.Thread(target=beside)
        t.start()
        t.join()
    assert not out, out
    torch.cuda.synchronize()
    assert same(img2, ref) and not same(img, ref)
    for _ in range(2):
        img.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert same(img, ref)
    ctx.check()
    ctx2.check()


@pytest.mark.parametrize("paths,spp", [(32, 3), (1700, 5), (1600, 4)])
def test_adjoint_in_several_launches(gpu_ctx, oracle_mod, limit, paths, spp):
    """33 x 17 pixels are 25 tiles, 800 paths a sample."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import RayTracer
    g, lb, alb, em = gi(gpu_ctx)
    cam, rt = scenes.gi_camera(33, 17), RayTracer(gpu_ctx)
    d_image = torch.rand(33 * 17, 4, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    limit("PATHS", paths)
    d_alb, d_le = rt.pathtrace_adjoint(lb, alb, em, cam, spp, 3, 9, d_image)
    gpu_ctx.check()
    nodes, ids, _, _ = oracle_mod.lbvh_build(g.tris, 14)
    ref_alb, ref_le = oracle_mod.pathtrace_adjoint(nodes, 14, ids, g.tris, g.albedo, g.emission, cam, spp, 3, 9,
                                                   d_image.cpu().numpy())
    # sums of at most 561 x spp x 4 products of a few roundings each, in any order
    scale = np.abs(ref_alb).max()
    assert np.abs(d_alb.cpu().numpy().astype(np.float64) - ref_alb).max() <= 1e-4 * scale
    assert np.allclose(d_le.cpu().numpy(), ref_le, rtol=1e-4, atol=1e-4 * np.abs(ref_le).max())


@pytest.mark.parametrize("held", [1, 1000, None])
def test_more_rays_in_doubt_than_listed(gpu_ctx, oracle_mod, limit, held):
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    from test_gpu_ray_calls import make_rays
    tris, depth, n = scenes.random_soup(20000, 10), 16, 700001
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    r = make_rays(tris, n)
    ref, st = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(*r), any_hit=True, stats=True)
    limit("RECHECKED_RAYS", held)
    gpu_ctx.set_trace_budget(40)
    got = hits_to_numpy(RayTracer(gpu_ctx).rays(lb, rays_tensor(*r, "cuda"), any_hit=True))
    gpu_ctx.check()
    assert np.array_equal(got["id"] >= 0, ref["id"] >= 0)
    within = st.sum(1) <= 40
    assert np.array_equal(got[within].view(np.int32), ref[within].view(np.int32))
    assert within.sum() > 1000 and (~within).sum() > 10000


def test_tree_without_records(gpu_ctx, oracle_mod, limit):
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    from test_gpu_ray_calls import make_rays
    from test_gpu_whitted import materials
    tris, depth = scenes.random_soup(20000, 10), 16
    dev = torch.from_numpy(tris).cuda()
    limit("TRACE_RECORDS", (32 << (depth - 1)) - 1)
    torch.cuda.synchronize()
    lb = LBVH(gpu_ctx, len(tris), depth)
    limit("TRACE_RECORDS", 32 << (depth - 1))
    with_records = LBVH(gpu_ctx, len(tris), depth)
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    rt = RayTracer(gpu_ctx)
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=183, height=97)
    light = (0.5, 3.0, 0.4)
    colour = torch.rand(len(tris), 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    out = []
    for tree in (lb, with_records):
        for how in (lambda: tree.Build(dev), lambda: tree.Import(nodes, ids, tris)):
            how()
            r = make_rays(tris, 20001)
            rays = rays_tensor(*r, "cuda")
            prim, leaves = rt.primary_leaves(tree, cam)
            res = [rt.rays(tree, rays), rt.rays(tree, rays[:999].contiguous()), *rt.rays_from(tree, rays, None), prim, leaves,
                   *rt.shadow_mirror_from(tree, cam, light, prim, leaves),
                   rt.whitted(tree, cam, light, materials(), bounces=2)[0],
                   rt.pathtrace(tree, colour, colour, cam, 2, 2, 5)]
            out.append([t.clone() for t in res])
            gpu_ctx.check()
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(*r))
    assert np.array_equal(hits_to_numpy(out[0][0]).view(np.int32), ref.view(np.int32))
    for o in out[1:]:
        for k, (a, b) in enumerate(zip(out[0], o)):
            if k not in (3, 5, 8):  # leaves: a handed-over ray reports the root
                assert torch.equal(a.view(torch.uint8), b.view(torch.uint8)), k


def test_batch_without_records(gpu_ctx, limit):
    import torch
    from rtgpu import scenes
    from rtgpu.api import Batch
    counts = [700, 1, 5000, 90]
    tris = torch.from_numpy(scenes.random_soup(sum(counts), 6, 0.02, 0.1)).cuda()
    cams, lights = scenes.batch_views(len(counts), 65, 49)
    got = []
    for size in (None, 0):
        limit("TRACE_RECORDS", size)
        b = Batch(gpu_ctx, counts, 14)
        b.set_views(cams, lights)
        hits, vis = b.alloc_outputs()
        b.build(tris)
        b.trace(hits, vis)
        alone = b.alloc_outputs(False)[0]
        b.trace(alone, None)
        gpu_ctx.check()
        assert torch.equal(alone, hits)
        got.append((hits.clone(), vis.clone()))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert len(got[0][1].unique()) >= 3


def test_two_streams_on_a_fresh_tree(oracle_mod, rt_lib):
    """Two contexts trace a tree at once whose records neither has made."""
    import torch
    from rtgpu import scenes
    from rtgpu.api import Context, LBVH, RayTracer, hits_to_numpy, rays_tensor
    from test_gpu_ray_calls import make_rays
    streams = [torch.cuda.Stream() for _ in range(3)]
    ctxs = [Context(0, s) for s in streams]
    n, depth = 60000, 18
    soups = [scenes.random_soup(n, 41), scenes.random_soup(n, 42)]
    dev = [torch.from_numpy(s).cuda() for s in soups]
    lb = LBVH(ctxs[0], n, depth)
    refs, rays = [], []
    for s in soups:
        nodes, ids, _, _ = oracle_mod.lbvh_build(s, depth)
        r = make_rays(s, 20000)
        rays.append(rays_tensor(*r, "cuda"))
        refs.append(oracle_mod.trace(nodes, depth, ids, s, oracle_mod.rays_array(*r)))
    rts = [RayTracer(c) for c in ctxs]
    torch.cuda.synchronize()
    for turn in range(6):
        k = turn % 2
        lb.Build(dev[k])
        built = streams[0].record_event()
        out = []
        for i in (1, 2):
            streams[i].wait_event(built)
            with torch.cuda.stream(streams[i]):
                out.append(rts[i].rays(lb, rays[k]))
        for s in streams[1:]:
            streams[0].wait_event(s.record_event())
        torch.cuda.synchronize()
        for o in out:
            assert np.array_equal(hits_to_numpy(o).view(np.int32), refs[k].view(np.int32)), turn
    for c in ctxs:
        c.check()
