"""Leaves over more emission tiles than a block or a warp looks back over at once: their start,
boxes and records, bit for bit against the oracle, in a tree and in a batch."""
import numpy as np
import pytest

from bitcmp import same_bits
from test_gpu_small_build import check

pytestmark = pytest.mark.gpu


def soup(runs, seed=4):
    """Runs of triangles with one code each and boxes of their own."""
    from rtgpu import scenes
    base = scenes.random_soup(len(runs), seed, 0.05, 0.2)
    tris = np.repeat(base, runs, 0).reshape(-1, 3, 3)
    tris += np.random.default_rng(seed).normal(0, 1e-7, tris.shape).astype(np.float32)
    return np.ascontiguousarray(tris.reshape(-1, 9))


@pytest.mark.parametrize("runs", [(17000, 5), (2047, 1, 16384, 3), (3, 2048, 2049), (512 * 33, 512 * 32 - 1, 2)])
def test_tree(gpu_ctx, oracle_mod, runs):
    from rtgpu.api import LBVH
    tris = soup(runs)
    check(gpu_ctx, oracle_mod, LBVH(gpu_ctx, len(tris), 12), tris, 12)


def test_batch(gpu_ctx, oracle_mod):
    import torch
    from rtgpu.api import Batch
    parts = [soup((400, 17000, 7), 1), soup((20000,), 2), soup((3, 9000, 9000), 3)]
    b = Batch(gpu_ctx, [len(p) for p in parts], 14).build(torch.from_numpy(np.concatenate(parts)).cuda())
    gpu_ctx.check()
    for s, p in enumerate(parts):
        nodes, ids, keys = b.download(s)
        onodes, oids, okeys, reached = oracle_mod.lbvh_build(p, 14)
        r = np.nonzero(reached)[0]
        assert np.array_equal(keys, okeys) and np.array_equal(ids, oids) and same_bits(nodes[r], onodes[r])


def test_memory_of_a_tree(gpu_ctx):
    """What a tree of 8 M triangles holds: 36 + 48 bytes of triangles, 16 of codes and ids and their
    alternates, 4 of leaves, and about 2 of the sort's and the emission's scratch each."""
    import torch
    from rtgpu.api import LBVH
    n = 8 << 20
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    lb = LBVH(gpu_ctx, n, 10)
    used = before - torch.cuda.mem_get_info()[0]
    lb.close()
    assert 104 * n < used < 108 * n
