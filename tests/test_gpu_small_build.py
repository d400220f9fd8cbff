"""The one-block build (k_build_small) at the edges of its warps, of its two
sizes and of its range, against the oracle: codes, permutation, reachable nodes
and sorted triangles bit for bit, and a trace through the records made from
it.  Beside soups: runs of equal codes (leaves above and below the size that a
warp folds), shallow heaps, and a larger build on the same handle before and
after."""
import numpy as np
import pytest

from bitcmp import same_bits

pytestmark = pytest.mark.gpu


def check(ctx, oracle_mod, lb, tris, depth):
    import torch
    from rtgpu import scenes
    from rtgpu.api import RayTracer, hits_to_numpy
    lb.Build(torch.from_numpy(tris).cuda())
    ctx.check()
    nodes, ids, keys = lb.download(True, True, True)
    onodes, oids, okeys, reached = oracle_mod.lbvh_build(tris, depth)
    assert np.array_equal(keys, okeys) and np.array_equal(ids, oids)
    r = np.nonzero(reached)[0]
    assert same_bits(nodes[r], onodes[r])
    cam = scenes.look_at((0.5, 0.8, -1.2), (0.5, 0.5, 0.5), width=61, height=37)
    hits = hits_to_numpy(RayTracer(ctx).primary(lb, cam))
    ref = oracle_mod.trace(onodes, depth, oids, tris, oracle_mod.primary_rays(cam))
    ctx.check()
    assert np.array_equal(hits.view(np.int32), ref.view(np.int32))


@pytest.mark.parametrize("n,depth", [(1, 1), (2, 1), (2, 20), (31, 9), (32, 3), (33, 20), (1023, 20), (1024, 12), (1025, 14),
                                     (2047, 20), (2048, 11), (2049, 14), (4095, 5), (4096, 20), (4097, 20)])
def test_soup(gpu_ctx, oracle_mod, n, depth):
    from rtgpu import scenes
    from rtgpu.api import LBVH
    check(gpu_ctx, oracle_mod, LBVH(gpu_ctx, n, depth), scenes.random_soup(n, n, 0.01, 0.2), depth)


@pytest.mark.parametrize("runs", [(4096,), (16, 17, 33, 700), (1,) * 40 + (2000,), (64,) * 64])
def test_equal_codes(gpu_ctx, oracle_mod, runs):
    from rtgpu import scenes
    from rtgpu.api import LBVH
    tris = np.repeat(scenes.random_soup(len(runs), 3, 0.05, 0.2), runs, 0)
    check(gpu_ctx, oracle_mod, LBVH(gpu_ctx, len(tris), 14), np.ascontiguousarray(tris), 14)


def test_handle_shared_with_the_general_build(gpu_ctx, oracle_mod):
    from rtgpu import scenes
    from rtgpu.api import LBVH
    lb = LBVH(gpu_ctx, 9000, 15)
    for n in (9000, 700, 5000, 4096, 3):
        check(gpu_ctx, oracle_mod, lb, scenes.random_soup(n, n + 1), 15)


@pytest.mark.parametrize("n,depth", [(4608, 20), (4609, 4), (155648, 20), (155649, 12), (1048576, 20), (1048577, 21),
                                     (1245184, 22), (1245185, 22)])
def test_tiles_of_the_general_build(gpu_ctx, oracle_mod, n, depth):
    """Around a whole emission tile and around the sizes where the sort changes
    its tile and the chunks their threads; the handle is larger than the soup."""
    from rtgpu import scenes
    from rtgpu.api import LBVH
    check(gpu_ctx, oracle_mod, LBVH(gpu_ctx, n + 300000, depth), scenes.random_soup(n, n, 0.001, 0.02), depth)


def test_long_leaves_across_tiles(gpu_ctx, oracle_mod):
    """Equal codes over several emission tiles, a leaf that ends at a tile's end and
    tiles inside one leaf."""
    from rtgpu import scenes
    from rtgpu.api import LBVH
    runs = (300, 212, 2048, 1, 3000, 511, 1, 600)
    tris = np.repeat(scenes.random_soup(len(runs), 4, 0.05, 0.2), runs, 0)
    check(gpu_ctx, oracle_mod, LBVH(gpu_ctx, len(tris), 14), np.ascontiguousarray(tris), 14)
