"""The dispatch of a caller's rays at the sizes where it changes: a warp per ray or a lane, a ray
for every lane of the GPU and one more, any-hit calls from which on the trace records are
walked, and restarted any-hit rays.  Half of the rays are ones that the records do not serve (along
an axis or a plane, from far away).  Hits are the oracle's on their bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(gpu_ctx, oracle_mod):
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH
    tris, depth = scenes.random_soup(20000, 10), 16
    lb = LBVH(gpu_ctx, len(tris), depth).Build(torch.from_numpy(tris).cuda())
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, depth)
    return tris, depth, lb, nodes, ids


def make_rays(tris, n):
    rng = np.random.default_rng(n)
    t = tris[rng.integers(0, len(tris), n)].reshape(n, 3, 3).mean(1)
    d = rng.normal(size=(n, 3))
    k = np.arange(n) % 6
    d[k == 0] *= [0, 0, 1]
    d[k == 1] *= [1, 0, 1]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = t - d * np.where(k == 2, 60.0, rng.uniform(0.0, 1.0, n))[:, None]
    tmax = np.where(np.arange(n) % 4 == 0, 0.3, 1e16)
    tmax[k == 2] = 1e16
    return o.astype(np.float32), d.astype(np.float32), tmax.astype(np.float32), np.full(n, -1, np.int32)


@pytest.mark.parametrize("n", [1, 33, 16384, 16385, "lanes", "lanes + 1"])
def test_closest(gpu_ctx, oracle_mod, scene, n):
    import torch
    from rtgpu.api import RayTracer, hits_to_numpy, rays_tensor
    tris, depth, lb, nodes, ids = scene
    if isinstance(n, str):
        n = torch.cuda.get_device_properties(0).multi_processor_count * 1024 + (1 if "+" in n else 0)
    r = make_rays(tris, n)
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(*r))
    got = hits_to_numpy(RayTracer(gpu_ctx).rays(lb, rays_tensor(*r, "cuda")))
    gpu_ctx.check()
    assert np.array_equal(got.view(np.int32), ref.view(np.int32))


@pytest.mark.parametrize("n", [699999, 700000])
@pytest.mark.parametrize("restart", [False, True])
def test_any_hit(gpu_ctx, oracle_mod, scene, n, restart):
    import torch
    from rtgpu.api import RayTracer, hits_to_numpy, rays_tensor
    tris, depth, lb, nodes, ids = scene
    r = make_rays(tris, n)
    rays = oracle_mod.rays_array(*r)
    starts = None
    if restart:
        _, starts = oracle_mod.trace_from(nodes, depth, ids, tris, rays)
    ref, _, st = oracle_mod.trace_from(nodes, depth, ids, tris, rays, starts, any_hit=True, stats=True)
    rt = RayTracer(gpu_ctx)
    t = rays_tensor(*r, "cuda")
    if restart:
        got, _ = rt.rays_from(lb, t, torch.from_numpy(starts.view(np.int32)).cuda(), any_hit=True)
    else:
        got = rt.rays(lb, t, any_hit=True)
    gpu_ctx.check()
    got = hits_to_numpy(got)
    assert np.array_equal(got["id"] >= 0, ref["id"] >= 0)
    within = st.sum(1) <= 384  # a ray over the budget reports some hit
    assert np.array_equal(got[within].view(np.int32), ref[within].view(np.int32)) and within.mean() > 0.5
