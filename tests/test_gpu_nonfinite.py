"""Soups with NaN vertices.  The build reports them, and the tree that it leaves is traced
as the oracle traces that tree: a box whose bounds are NaN along an axis is entered
whatever the ray does there, so no other triangle is lost.  Imported trees whose boxes
hold their bounds in the other order are traced as the oracle does too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def traced(ctx, oracle_mod, lb, nodes, depth, ids, tris, seed):
    from rtgpu import scenes
    from rtgpu.api import RayTracer, hits_to_numpy, rays_tensor
    rt = RayTracer(ctx)
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=320, height=200)
    rng = np.random.default_rng(seed)
    n = 20000
    o = rng.uniform(-1, 2, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    args = (o, d, np.full(n, 1e16, np.float32), np.full(n, -1, np.int32))
    prim, ref = hits_to_numpy(rt.primary(lb, cam)), oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.primary_rays(cam))
    rays, rref = hits_to_numpy(rt.rays_from(lb, rays_tensor(*args, "cuda"), None)[0]), oracle_mod.trace(
        nodes, depth, ids, tris, oracle_mod.rays_array(*args))
    assert np.array_equal(prim.view(np.int32), ref.view(np.int32))
    assert np.array_equal(rays.view(np.int32), rref.view(np.int32))
    assert (ref["id"] >= 0).mean() > 0.2


@pytest.mark.parametrize("n", [1500, 6000])
@pytest.mark.parametrize("vertex,axis", [(0, 0), (0, 1), (0, 2), (1, 1), (2, 0)])
def test_nan_vertices(gpu_ctx, oracle_mod, n, vertex, axis):
    import torch
    from rtgpu import scenes
    from rtgpu._lib import RtError
    from rtgpu.api import LBVH
    tris = scenes.random_soup(n, 12, 0.02, 0.1)
    tris[np.random.default_rng(1).integers(0, n, 40), 3 * vertex + axis] = np.nan
    lb = LBVH(gpu_ctx, n, 16).Build(torch.from_numpy(tris).cuda())
    with pytest.raises(RtError, match="NaN or Inf"):
        gpu_ctx.check()
    nodes, ids, _ = lb.download(True, True)
    traced(gpu_ctx, oracle_mod, lb, nodes, 16, ids, tris, 3)
    gpu_ctx.check()


def test_bounds_in_the_other_order(gpu_ctx, oracle_mod):
    from rtgpu import scenes
    from rtgpu.api import LBVH
    tris = scenes.random_soup(6000, 13, 0.02, 0.1)
    nodes, ids, _, reached = oracle_mod.lbvh_build(tris, 16)
    turn = np.random.default_rng(2).random((len(nodes), 3)) < 0.5
    turn[1] = False
    lo, hi = nodes["min"].copy(), nodes["max"].copy()
    nodes["min"], nodes["max"] = np.where(turn, hi, lo), np.where(turn, lo, hi)
    lb = LBVH(gpu_ctx, len(tris), 16).Import(nodes, ids, tris)
    traced(gpu_ctx, oracle_mod, lb, nodes, 16, ids, tris, 4)
    gpu_ctx.check()
