"""The emitter gradient of the adjoint is the sum over all paths rounded once: with no
bounce, one or two samples and a whole-number image gradient every path's term is exact in 32 bits (whole
numbers below 2^12 times a power of two), as are the few that a lane adds up; the total is not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp,paths", [(8, 4, 1, None), (128, 96, 1, None), (301, 203, 2, None), (512, 512, 2, None),
                                           (300, 203, 2, 64 * 1024), (128, 96, 2, 32)])
def test_sum_over_all_paths_is_rounded_once(gpu_ctx, w, h, spp, paths):
    import torch
    from rtgpu import _lib as L
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer
    g = scenes.gi_box(200, seed=4)
    lb = LBVH(gpu_ctx, len(g.tris), 12).Build(torch.from_numpy(g.tris).cuda())
    emission = torch.full((len(g.tris), 3), 2.0, device="cuda")  # every triangle emits
    albedo = torch.from_numpy(g.albedo).cuda()
    cam, rt = scenes.gi_camera(w, h), RayTracer(gpu_ctx)
    # a pixel's mean counts the samples that hit: all paths end at their first hit
    seen = rt.pathtrace(lb, albedo, emission, cam, spp, 0, 5, sky=(0.0, 0.0, 0.0)).cpu().numpy()[:, :3].astype(np.float64) / 2.0
    assert seen.max() == 1.0
    rng = np.random.default_rng(8)
    d = np.zeros((w * h, 4), np.float32)
    d[:, :3] = rng.integers(0, 1 << 12, (w * h, 3))
    gpu_ctx.set_limit(L.RT_LIMIT_PATHS, paths)
    try:
        _, got = rt.pathtrace_adjoint(lb, albedo, emission, cam, spp, 0, 5, torch.from_numpy(d).cuda(), sky=(0.0, 0.0, 0.0))
        gpu_ctx.check()
    finally:
        gpu_ctx.set_limit(L.RT_LIMIT_PATHS, None)
    exact = (seen * d[:, :3]).sum(0)  # whole multiples of 1 / spp below 2^32: exact in 64 bits
    assert np.array_equal(got.cpu().numpy(), exact.astype(np.float32)), (got, exact)
