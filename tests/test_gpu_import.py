"""Imported trees (rt_lbvh_import_host), which the caller made: leaves whose triangle range
is not the tree's and ids past the soup end in the bounds error and are not read; trees
that no build makes, with empty leaves and with several leaves over the same triangles,
are traced as the oracle traces them, to the bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, DEPTH = 5000, 14


def made(oracle_mod, seed=31):
    from rtgpu import scenes
    tris = scenes.random_soup(N, seed, 0.02, 0.1)
    nodes, ids, _, _ = oracle_mod.lbvh_build(tris, DEPTH)
    return tris, nodes, ids


def reached_leaves(nodes):
    out, todo = [], [1]
    while todo:
        h = todo.pop()
        if int(nodes[h]["prim_count"]) & 4:
            out.append(h)
        else:
            todo += [2 * h, 2 * h + 1]
    return out


def rays_at(tris, n, seed=3):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-1, 2, (n, 3)).astype(np.float32)
    d = tris[rng.integers(0, len(tris), n), :3] - o
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    return o, d, np.full(n, 1e16, np.float32), np.full(n, -1, np.int32)


@pytest.mark.parametrize("pos,count", [(-1, 40), (-1, 2), (-2**31, 31), (N - 39, 40), (N, 1), (0, -1), (100, -2**20), (7, N)])
def test_leaf_out_of_range(gpu_ctx, oracle_mod, pos, count):
    import torch
    from rtgpu import scenes
    from rtgpu._lib import RtError
    from rtgpu.api import LBVH, RayTracer, rays_tensor
    from test_gpu_whitted import materials
    tris, nodes, ids = made(oracle_mod)
    for h in reached_leaves(nodes):
        nodes[h]["prim_pos"] = pos
        nodes[h]["prim_count"] = (count << 3) | (int(nodes[h]["prim_count"]) & 7)
    lb = LBVH(gpu_ctx, N, DEPTH).Import(nodes, ids, tris)
    rt = RayTracer(gpu_ctx)
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=160, height=96)
    rays = rays_tensor(*rays_at(tris, 20000), "cuda")
    colour = torch.full((N, 3), 0.5, device="cuda")

    def refused(call):
        call()
        with pytest.raises(RtError, match="bounds check"):
            gpu_ctx.check()

    refused(lambda: rt.primary(lb, cam))
    refused(lambda: rt.rays(lb, rays))
    refused(lambda: rt.rays_from(lb, rays, None))
    refused(lambda: rt.rays(lb, rays, any_hit=True))
    refused(lambda: rt.whitted(lb, cam, (0.5, 3.0, 0.4), materials(), bounces=0))
    refused(lambda: rt.pathtrace(lb, colour, colour, cam, 2, 1, 5))
    gpu_ctx.check()  # the error was cleared


@pytest.mark.parametrize("bad", [N, 2**31, 2**32 - 1])
def test_id_out_of_range(gpu_ctx, oracle_mod, bad):
    from rtgpu._lib import RtError
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris, nodes, ids = made(oracle_mod)
    wrong = ids.copy()
    wrong[[0, 77, N - 1]] = bad
    lb = LBVH(gpu_ctx, N, DEPTH).Import(nodes, wrong, tris)
    with pytest.raises(RtError, match="bounds check"):
        gpu_ctx.check()
    hits = hits_to_numpy(RayTracer(gpu_ctx).rays(lb, rays_tensor(*rays_at(tris, 20000), "cuda")))
    gpu_ctx.check()
    assert hits["id"].min() >= -1 and hits["id"].max() < N
    lb.Import(nodes, ids, tris)  # the handle still serves
    gpu_ctx.check()


def split_leaves(nodes, depth, how):
    """Every leaf becomes an internal node: of it and an empty leaf at the same position (right
    or left), or of two leaves over the same triangles, one per half of the box."""
    out = np.zeros(1 << depth, nodes.dtype)
    out[:len(nodes)] = nodes
    for h in reached_leaves(nodes):
        leaf = nodes[h]
        l, r = leaf.copy(), leaf.copy()
        if how == "shared":
            a = int(np.argmax(leaf["max"] - leaf["min"]))
            l["max"][a] = r["min"][a] = np.float32(0.5) * (leaf["min"][a] + leaf["max"][a])
        else:
            e = r if how == "empty right" else l
            e["prim_count"] = 4
            e["max"] = e["min"]
        out[2 * h], out[2 * h + 1] = l, r
        out[h]["prim_count"] = (int(leaf["prim_count"]) >> 3) << 3 | 1
    return out


@pytest.mark.parametrize("how", ["empty right", "empty left", "shared"])
def test_leaves_at_one_position(gpu_ctx, oracle_mod, how):
    import torch
    from rtgpu import scenes
    from rtgpu.api import LBVH, RayTracer, hits_to_numpy, rays_tensor
    tris, nodes, ids = made(oracle_mod)
    depth = DEPTH + 1
    nodes = split_leaves(nodes, depth, how)
    lb = LBVH(gpu_ctx, N, depth).Import(nodes, ids, tris)
    rt = RayTracer(gpu_ctx)
    o, d, tmax, excl = rays_at(tris, 40000)
    d[::5, 2] = 0.0  # rays that the trace records do not serve
    ref = oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.rays_array(o, d, tmax, excl))
    rays = rays_tensor(o, d, tmax, excl, "cuda")
    got, leaves = rt.rays_from(lb, rays, None)
    again, _ = rt.rays_from(lb, rays, leaves)
    few = rt.rays(lb, rays[:5000].contiguous())
    cam = scenes.look_at((1.7, 1.2, 1.5), (0.5, 0.5, 0.5), vfov_deg=45.0, width=161, height=97)
    prim = rt.primary(lb, cam)
    gpu_ctx.check()
    same = lambda a, b: np.array_equal(hits_to_numpy(a).view(np.int32), b.view(np.int32))  # noqa: E731
    assert same(got, ref) and same(again, ref) and same(few, ref[:5000])
    assert same(prim, oracle_mod.trace(nodes, depth, ids, tris, oracle_mod.primary_rays(cam)))
    hit = ref["id"] >= 0
    slots = leaves.cpu().numpy()
    assert hit.mean() > 0.2 and (slots[~hit] == 1).all()
    hit &= slots != 1  # a handed-over ray reports the root
    assert hit.mean() > 0.2
    pc, pos = nodes["prim_count"][slots[hit]], nodes["prim_pos"][slots[hit]]
    where = np.empty(N, np.int64)
    where[ids] = np.arange(N)
    at = where[ref["id"][hit]]
    assert (pc & 4).all() and ((pos <= at) & (at < pos + (pc >> 3))).all()
