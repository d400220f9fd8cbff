// rt_trace.cu -- primary, shadow and mirror rays over the LBVH on sm_103a.
//
// Replaces the per-bounce dispatches of RayTracerCS::Render
// (RayTracerCS/RayTracerCS.cpp:284-295): CSGeneratePrimaryRays
// (Shaders/CS/CSPrimaryRays.hlsl:22-69) and CSComputeIntersections
// (CSIntersections.hlsl:18-39) are fused into k_walk_primary (rays are made
// in registers, no 48-byte ray buffer round trip); the shadow ray and the
// mirror bounce of CSComputeColor (CSComputeColorRT.hlsl:57-177, 203-210,
// flat normals, no textures) are k_walk_shade; a caller's own rays are
// k_walk_rays.  All three walk the trace records (Walk in rt_traverse.cuh).
// k_trace_primary, k_trace_secondary and k_trace_rays walk the heap and count
// every box and triangle test.
//
// The kernels are persistent: a grid sized to fill every SM once, each
// warp pulling 32-ray tiles (8 x 4 pixels) or single rays from a work counter
// until the image is done.  Ray cost varies by three orders of magnitude across
// the image, so a static grid leaves SMs idle behind the last heavy tiles.
#include <algorithm>
#include <cstring>
#include <initializer_list>

#include "rt_records.cuh"
#include "rt_traverse.cuh"

using namespace rt;

namespace {

constexpr int kTraceThreads = 128;

__device__ __forceinline__ void store_hit(rt_hit* out, const Hit& h) {
    *reinterpret_cast<int4*>(out) = make_int4(h.id, __float_as_int(h.u), __float_as_int(h.v), __float_as_int(h.t));
}

// Heavy-ray list entries: kind in the top two bits, pixel or ray index below.
enum : uint32_t { kHeavyPrimary = 0, kHeavyShadow = 1, kHeavyMirror = 2, kHeavyRay = 3 };
constexpr uint32_t kHeavyIndexMask = (1u << 30) - 1u;

__device__ __forceinline__ void spill_record(uint32_t* list, int slot, uint32_t kind, size_t index) {
    list[slot] = (kind << 30) | (uint32_t)index;
}

constexpr uint32_t kNoSlot = 0xffffffffu;

// Warp-aggregated append of the lanes' pixels to a list (a warp's pixels in
// lane order, so neighbouring rays stay neighbours).  Returns the lane's
// slot, or kNoSlot.
__device__ __forceinline__ uint32_t append_pixel(bool take, uint32_t p, uint32_t* list, uint32_t cap,
                                                 uint32_t* count) {
    const uint32_t m = __ballot_sync(0xffffffffu, take);
    if (!m) return kNoSlot;
    uint32_t base = 0;
    if ((threadIdx.x & 31) == 0) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t k = base + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
    if (!take || k >= cap) return kNoSlot;
    list[k] = p;
    return k;
}

// The shading-ray lists of a frame (shadow pixels, then mirror pixels) and
// the results that need no ray.  A frame's primary pass fills them as it
// goes (lists != nullptr), so no separate pass re-reads the primary hits.
// Beside each listed pixel its ray (two float4: origin and tmax, direction
// and the excluded triangle) and the node its walk starts at, so the
// tracing kernel neither re-reads the primary hit and the triangle nor
// rebuilds the ray.
struct ShadeLists {
    const float* soup;
    float lx, ly, lz;
    uint8_t* vis;
    rt_hit* mirror;
    uint32_t* lists;
    uint32_t cap;
    uint32_t* counts;  // 2 words
    float4* rays;      // 2 x cap rays (2 float4 each), by list slot
    uint32_t* starts;  // 2 x cap start nodes, by list slot
};

__device__ __forceinline__ void put_ray(float4* q, const RayState& r) {
    q[0] = make_float4(r.o.x, r.o.y, r.o.z, r.tmax);
    q[1] = make_float4(r.d.x, r.d.y, r.d.z, __int_as_float(r.exclude));
}

// One pixel's shading-ray setup from its primary hit ph (all lanes call):
// visibility 0 (no hit) or 1 (light behind the surface) and the mirror
// miss record are written, the pixels that cast a shadow ray and those that
// cast a mirror ray are appended to the two lists with their rays and
// `start`, the restart node of the walks (the primary hit's leaf, or 1).
__device__ __forceinline__ void shade_setup_pixel(const ShadeLists& sl, const rt_camera& cam, int4 ph, bool valid,
                                                  uint32_t i, uint32_t j, size_t p, uint32_t start) {
    const ShadeRays s = shade_rays(sl.soup, cam, sl.lx, sl.ly, sl.lz, ph, valid, i, j, sl.mirror != nullptr);
    if (valid) {
        if (sl.vis && !(s.has && s.cast)) sl.vis[p] = vis_code(s.has, s.cast, false);
        if (sl.mirror && !s.has) {
            Hit mh;
            mh.id = -2; mh.u = -1.0f; mh.v = -1.0f; mh.t = 0.0f;
            store_hit(sl.mirror + p, mh);
        }
    }
    const uint32_t ks = append_pixel(sl.vis && valid && s.has && s.cast, (uint32_t)p, sl.lists, sl.cap, sl.counts);
    const uint32_t km = append_pixel(sl.mirror && valid && s.has, (uint32_t)p, sl.lists + sl.cap, sl.cap, sl.counts + 1);
    if (ks != kNoSlot) {
        put_ray(sl.rays + 2 * (size_t)ks, s.shadow);
        sl.starts[ks] = start;
    }
    if (km != kNoSlot) {
        put_ray(sl.rays + 2 * ((size_t)sl.cap + km), s.mirror);
        sl.starts[sl.cap + km] = start;
    }
}

// Primary rays with their box and triangle test counts, in the oracle's order.
__global__ void __launch_bounds__(kTraceThreads, 7) k_trace_primary(TreeRef tr, rt_camera cam,
                                                                    rt_hit* __restrict__ hits,
                                                                    uint32_t* __restrict__ leaves,
                                                                    uint32_t* __restrict__ stats, uint32_t* work,
                                                                    uint32_t num_tiles, TileOrder ord) {
    const uint32_t wbuf = *ord.parity, rbuf = wbuf ^ 1u, heavy = min(ord.counts[rbuf], ord.cap);
    for (uint32_t tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles); tile < num_tiles;
         tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles)) {
        uint32_t i, j;
        const bool valid = tile_pixel(tile, threadIdx.x & 31, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;  // lanes past the image edge only help the warp
        const RayState r = make_ray(mk3(cam.eye[0], cam.eye[1], cam.eye[2]), primary_dir(cam, i, j), 1e16f, -1);
        uint32_t nb = 0, nt = 0, leaf = 1;
        const Hit h = trace_ray<true>(r, valid, tr, false, &nb, &nt, nullptr, nullptr, 1u, &leaf);
        if (valid) {
            const size_t p = (size_t)j * cam.width + i;
            store_hit(hits + p, h);
            if (leaves) leaves[p] = leaf;
            stats[2 * p] = nb;
            stats[2 * p + 1] = nt;
        }
        record_tile_cost(ord, wbuf, tile, nb + nt);
    }
}

// Primary rays over the trace records (Walk), an 8 x 4 tile per warp at a time:
// neighbouring rays visit the same leaves, so handing out pixels one by one to the
// lanes that are done (as the shading rays are) was slower.
// Of kPrimSteps 3, 4 and 8: 1,415, 1,423 and 1,413 us a frame of 2.1 M triangles at
// 1080p, 312, 309 and 330 us of 65 k triangles at 512 x 512.
constexpr int kPrimSteps = 3;

// Blocks per SM: with few tiles a warp the image lasts as long as its slowest tiles,
// and 72 registers (no spills) move a lane faster; with many, 64 registers and
// another block per SM hide more latency (65 k triangles at 512 x 512 275 us a frame with
// eight blocks and 272 with seven, 260 k at 720p 583 and 576, 2.1 M at 1080p
// 1,404 and 1,412).
constexpr uint32_t kPrimWarps = 8u * kTraceThreads / 32u;  // warps an SM
uint32_t prim_blocks(const rt_ctx* ctx, uint32_t tiles) {
    return tiles > 8u * kPrimWarps * (uint32_t)ctx->num_sms ? 8u : 7u;
}

template <int BLOCKS>
__global__ void __launch_bounds__(kTraceThreads, BLOCKS) k_walk_primary(TreeRef tr, rt_camera cam,
                                                                        rt_hit* __restrict__ hits,
                                                                        uint32_t* __restrict__ leaves, uint32_t* work,
                                                                        uint32_t num_tiles, Spill spill,
                                                                        uint32_t* __restrict__ list, TileOrder ord,
                                                                        ShadeLists sl) {
    constexpr uint32_t kFull = 0xffffffffu;
    grid_dep_wait();
    mark_records(tr);
    const uint32_t wbuf = *ord.parity, rbuf = wbuf ^ 1u, heavy = min(ord.counts[rbuf], ord.cap);
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    bool budgeted = spill.count != nullptr;
    for (uint32_t tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles); tile < num_tiles;
         tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles)) {
        uint32_t i, j;
        const bool valid = tile_pixel(tile, threadIdx.x & 31, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;  // lanes past the image edge only help the warp
        int slot = -1;
        w.tests = 0u;
        const RayState r = make_ray(mk3(cam.eye[0], cam.eye[1], cam.eye[2]), primary_dir(cam, i, j), 1e16f, -1);
        w.start(valid, r, tr, 1u, stack, Walk::tile_by_heap(valid, r, tr));
        while (__any_sync(kFull, w.have)) {
            w.round(tr, kPrimSteps, stack);
            if (w.have && budgeted && w.tests > spill.budget) {
                const uint32_t e = atomicAdd(spill.count, 1u);
                if (e < spill.cap) {
                    slot = (int)e;
                    w.stop();
                } else {
                    budgeted = false;  // list full: finish here
                }
            }
        }
        const size_t p = (size_t)j * cam.width + i;
        const uint32_t leaf = tr.compact ? 1u : w.b.leaf;
        const Hit h = w.hit();
        if (valid) {
            store_hit(hits + p, h);  // of a handed-over ray: the closest hit so far
            if (slot >= 0) spill_record(list, slot, kHeavyPrimary, p);
            if (leaves) leaves[p] = leaf;
        }
        if (sl.lists) {  // uniform; a handed-over pixel is set up by the warp-per-ray pass
            const int4 ph = make_int4(h.id, __float_as_int(h.u), __float_as_int(h.v), __float_as_int(h.t));
            shade_setup_pixel(sl, cam, ph, valid && slot < 0, i, j, p, leaf);
        }
        record_tile_cost(ord, wbuf, tile, w.tests);
    }
}

// Restart node of a pixel's shading rays: its primary hit's leaf, or the root.
__device__ __forceinline__ uint32_t shade_start(const uint32_t* __restrict__ prim_leaves, int4 ph, bool valid,
                                                size_t p) {
    return (prim_leaves && valid && ph.x >= 0) ? __ldg(prim_leaves + p) : 1u;
}

// Shadow (any hit) and mirror (closest hit) rays with their test counts, in the
// oracle's order.  Rays of pixels whose primary ray missed, or whose light is
// behind the surface, are traced with active == false.
__global__ void __launch_bounds__(kTraceThreads) k_trace_secondary(
    TreeRef tr, const float* __restrict__ soup, rt_camera cam, float lx, float ly, float lz,
    const rt_hit* __restrict__ prim, const uint32_t* __restrict__ prim_leaves, uint8_t* __restrict__ vis,
    rt_hit* __restrict__ mirror, uint32_t* __restrict__ mirror_leaves, uint32_t* __restrict__ sstats,
    uint32_t* __restrict__ mstats, uint32_t* work, uint32_t num_tiles, TileOrder ord) {
    const uint32_t wbuf = *ord.parity, rbuf = wbuf ^ 1u, heavy = min(ord.counts[rbuf], ord.cap);
    for (uint32_t tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles); tile < num_tiles;
         tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles)) {
        uint32_t i, j;
        const bool valid = tile_pixel(tile, threadIdx.x & 31, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;  // lanes past the image edge only help the warp
        const size_t p = (size_t)j * cam.width + i;
        int4 ph = make_int4(-1, 0, 0, 0);
        if (valid) ph = __ldg(reinterpret_cast<const int4*>(prim + p));
        const uint32_t start = shade_start(prim_leaves, ph, valid, p);
        const ShadeRays s = shade_rays(soup, cam, lx, ly, lz, ph, valid, i, j, mirror != nullptr);
        uint32_t snb = 0, snt = 0, mnb = 0, mnt = 0;
        if (vis) {  // uniform across the warp
            const Hit sh = trace_ray<true>(s.shadow, s.cast, tr, true, &snb, &snt, nullptr, nullptr, start);
            if (valid) vis[p] = vis_code(s.has, s.cast, sh.id >= 0);
        }
        if (mirror) {
            uint32_t leaf = 1;
            Hit mh = trace_ray<true>(s.mirror, s.has, tr, false, &mnb, &mnt, nullptr, nullptr, start, &leaf);
            if (!s.has) {
                mh.id = -2; mh.u = -1.0f; mh.v = -1.0f; mh.t = 0.0f;
            }
            if (valid) {
                store_hit(mirror + p, mh);
                if (mirror_leaves) mirror_leaves[p] = leaf;
            }
        }
        if (valid) {
            if (sstats) { sstats[2 * p] = snb; sstats[2 * p + 1] = snt; }
            if (mstats) { mstats[2 * p] = mnb; mstats[2 * p + 1] = mnt; }
        }
        record_tile_cost(ord, wbuf, tile, snb + snt + mnb + mnt);
    }
}

// Production path of the shading rays, in two passes.  k_shade_setup runs
// over the pixels in 8x4-tile order, writes the results that need no ray (no
// primary hit: visibility 0 and the mirror miss record; light behind the
// surface: visibility 1) and appends the pixels that cast a shadow ray and
// those that cast a mirror ray to two lists, a warp's pixels in order, so
// neighbouring rays stay neighbours, each with the ray that k_trace_secondary
// would cast and its start node.  k_walk_shade then traces the lists with every
// lane busy (a pass over the pixels leaves the lanes of sky pixels and of
// pixels without a cast ray idle).
__global__ void __launch_bounds__(256) k_shade_setup(const float* __restrict__ soup, rt_camera cam, float lx, float ly,
                                                     float lz, const rt_hit* __restrict__ prim, uint8_t* __restrict__ vis,
                                                     rt_hit* __restrict__ mirror, uint32_t* __restrict__ mirror_leaves,
                                                     const uint32_t* __restrict__ prim_leaves,
                                                     uint32_t* __restrict__ lists, uint32_t cap, uint32_t* counts,
                                                     float4* __restrict__ rays, uint32_t* __restrict__ starts,
                                                     uint32_t num_tiles) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nwarps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t t = warp; t < num_tiles; t += nwarps) {
        uint32_t i, j;
        const bool valid = tile_pixel(t, lane, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;
        const size_t p = (size_t)j * cam.width + i;
        int4 ph = make_int4(-1, 0, 0, 0);
        if (valid) ph = __ldg(reinterpret_cast<const int4*>(prim + p));
        const ShadeLists sl{soup, lx, ly, lz, vis, mirror, lists, cap, counts, rays, starts};
        shade_setup_pixel(sl, cam, ph, valid, i, j, p, shade_start(prim_leaves, ph, valid, p));
        if (valid && mirror_leaves && ph.x < 0) mirror_leaves[p] = 1u;
    }
}

__device__ __forceinline__ RayState load_ray(const rt_ray* __restrict__ rays, uint32_t k, bool valid) {
    float4 a = make_float4(0.f, 0.f, 0.f, __int_as_float(-1)), b = make_float4(0.f, 0.f, 1.f, 1.f);
    if (valid) {
        a = __ldg(reinterpret_cast<const float4*>(rays + k));
        b = __ldg(reinterpret_cast<const float4*>(rays + k) + 1);
    }
    return make_ray(mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), b.w, __float_as_int(a.w));
}

// The shading pass keeps every lane busy: a lane whose ray has finished takes the
// next list entry once kWalkRefill lanes of its warp are idle (the newcomers
// take consecutive entries, so they stay neighbours), instead of idling until
// the warp's slowest ray is done (dynamic ray fetch, Aila and Laine 2009).
//
// It walks the trace records (Walk).  BATCH: a listed pixel g belongs to
// scene g / px, and a warp's lanes may walk different scenes.
// 16 idle lanes and 4 expansions a round were the fastest of 12 to 24 and 3 to 10:
// 650 -> 545 us a frame of 2.1 M triangles at 1080p.  A frame's rays take 72 registers
// (seven blocks an SM; five to eight at 260 k triangles and 720p: 570, 561, 555 and 565 us,
// at 2.1 M and 1080p 1,509, 1,446, 1,410 and 1,404), a batch's many scenes 64.
constexpr int kWalkRefill = 16;
constexpr int kWalkSteps = 4;
// A caller's rays: of 8 to 16 idle lanes, and 3 to 12 expansions a round.  A call that
// gives each lane one ray lasts as long as its longest chain of rounds, and a ray that reads the
// heap needs more of each: 20,000 rays from 60 extents away over 65 k triangles 228 us with
// 8 expansions, 220 with 6, 183 with 4, near ones 170, 168 and 169.  Many rays: 2^20 near ones over a
// soup 897, 890 and 957 us, along an axis 862, 834 and 889.
constexpr int kRayRefill = 8;
constexpr int kRaySteps = 6;
constexpr int kFewSteps = 4;
constexpr uint32_t kRayBlocks = 8u;
uint32_t ray_lanes(const rt_ctx* ctx) { return kRayBlocks * kTraceThreads * (uint32_t)ctx->num_sms; }

// The scenes of a batch.
struct BatchTrees {
    const rt_node* nodes;
    const TraceNode* tnodes;
    const uint32_t* tri_off;
    uint32_t depth, px;
};

__device__ __forceinline__ void scene_tree(TreeRef& tr, const BatchTrees& bt, uint32_t sc) {
    tr.heap = bt.nodes + ((size_t)sc << bt.depth);
    if (bt.tnodes) tr.tnodes = bt.tnodes + ((size_t)sc << (bt.depth - 1u));
    tr.tri_base = __ldg(bt.tri_off + sc);
    tr.n = __ldg(bt.tri_off + sc + 1);
}

template <bool BATCH>
__global__ void __launch_bounds__(kTraceThreads, BATCH ? 8 : 7) k_walk_shade(
    TreeRef tr0, uint8_t* __restrict__ vis, rt_hit* __restrict__ mirror, uint32_t* __restrict__ mirror_leaves,
    const uint32_t* __restrict__ lists, uint32_t cap, const uint32_t* counts, const float4* __restrict__ rays,
    const uint32_t* __restrict__ starts, uint32_t* work, Spill spill, uint32_t* __restrict__ list,
    BatchTrees bt) {
    constexpr uint32_t kFull = 0xffffffffu;
    grid_dep_wait();
    mark_records(tr0);
    TreeRef tr = tr0;
    const uint32_t ns = min(counts[0], cap), nm = min(counts[1], cap), total = ns + nm;
    const int lane = threadIdx.x & 31;
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    uint32_t p = 0;
    bool live = false, shadow = false, budgeted = spill.count != nullptr, drained = false;
    for (;;) {
        const uint32_t idle = __ballot_sync(kFull, !live);
        if (!drained && (idle == kFull || __popc(idle) >= kWalkRefill)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, (uint32_t)__popc(idle));
            base = __shfl_sync(kFull, base, 0);
            if (base + (uint32_t)__popc(idle) >= total) drained = true;
            const uint32_t k = base + __popc(idle & ((1u << lane) - 1u));
            const bool take = !live && k < total;
            RayState r = make_ray(mk3(0.f, 0.f, 0.f), mk3(0.f, 0.f, 1.f), 1.0f, -1);
            uint32_t start = 1u;
            if (take) {
                shadow = k < ns;
                const uint32_t q = shadow ? k : cap + (k - ns);  // list slot: pixel, ray, start node
                p = __ldg(lists + q);
                if (BATCH) scene_tree(tr, bt, p / bt.px);
                const float4 ra = __ldg(rays + 2 * (size_t)q), rb = __ldg(rays + 2 * (size_t)q + 1);
                r = make_ray(mk3(ra.x, ra.y, ra.z), mk3(rb.x, rb.y, rb.z), ra.w, __float_as_int(rb.w));
                start = __ldg(starts + q);
                live = true;
            }
            w.start(take, r, tr, start, stack);
        }
        if (!__any_sync(kFull, live)) {
            if (drained) break;
            continue;
        }
        w.round<kPoolMin, !BATCH>(tr, kWalkSteps, stack, shadow);
        int slot = -1;
        if (live && w.have && budgeted && w.tests > spill.budget) {
            const uint32_t e = atomicAdd(spill.count, 1u);
            if (e < spill.cap) {
                slot = (int)e;
                w.stop();
            } else {
                budgeted = false;  // list full: finish here
            }
        }
        if (live && !w.have) {  // the walk is over: the ray's result
            if (slot >= 0) spill_record(list, slot, shadow ? kHeavyShadow : kHeavyMirror, p);
            if (!shadow) {
                store_hit(mirror + p, w.hit());  // of a handed-over ray: the closest hit so far
                if (mirror_leaves) mirror_leaves[p] = tr.compact ? 1u : w.b.leaf;
            } else if (slot < 0) {
                vis[p] = vis_code(true, true, w.b.id >= 0);
            }
            live = false;
        }
    }
}

// Any-hit calls of fewer rays stay with traverse(): the second walk of the rays in
// doubt lasts as long as its longest ones, 150 us on a mesh's grazing rays, whatever
// their number.  Where the record walk becomes the faster one (us, traverse() and records):
// rays at a torus of 65 k triangles from around it 500,000 (448, 446), along planes through it
// 700,000 (555, 553); at 260 k triangles 460,000, and along planes 680,000; in a soup 150,000;
// short rays everywhere from the first thousand.  At 700,000 no kind is slower but rays along an
// axis of the 260 k triangles (232, 249; 4 M: 848, 989).  Restarted rays often end in their first
// leaf, and the second walk is then most of the call (2^20: 256, 470; rays that go on 782, 692).
constexpr uint32_t kWalkAnyRays = 700000u;

// The any-hit rays in doubt: their list, or, when more than `cap` are, the marks that
// each of them has left in its hit.
struct Doubt {
    uint32_t* list;
    uint32_t* count;
    uint32_t* work;
    uint32_t cap;
};
constexpr int kDoubtMark = -3;

// A caller's rays over the trace records.  A closest hit does not depend on the
// walk, so a ray over the budget goes to the warp-per-ray pass.  The first
// hit does: this walk meets the leaves in traverse()'s order, but which rays
// traverse() hands over depends on its exact counts, which are at most the
// counts here.  So an any-hit ray over the budget is walked again by
// k_trace_doubt, as traverse() does, with its budget.
template <int STEPS>
__global__ void __launch_bounds__(kTraceThreads, kRayBlocks) k_walk_rays(TreeRef tr, const rt_ray* __restrict__ rays, uint32_t n,
                                                                     int any_hit, const uint32_t* __restrict__ starts,
                                                                     rt_hit* __restrict__ hits,
                                                                     uint32_t* __restrict__ leaves, uint32_t* work,
                                                                     Spill spill, uint32_t* __restrict__ list, Doubt doubt) {
    constexpr uint32_t kFull = 0xffffffffu;
    grid_dep_wait();
    mark_records(tr);
    const int lane = threadIdx.x & 31;
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    uint32_t k = 0;
    bool live = false, budgeted = spill.count != nullptr, drained = false;
    for (;;) {
        const uint32_t idle = __ballot_sync(kFull, !live);
        if (!drained && (idle == kFull || __popc(idle) >= kRayRefill)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, (uint32_t)__popc(idle));
            base = __shfl_sync(kFull, base, 0);
            if (base >= n || n - base <= (uint32_t)__popc(idle)) drained = true;
            const uint32_t q = base + __popc(idle & ((1u << lane) - 1u));
            const bool take = !live && base < n && q < n;
            if (take) {
                k = q;
                live = true;
            }
            w.start(take, load_ray(rays, k, take), tr, (starts && take) ? __ldg(starts + k) : 1u, stack);
        }
        if (!__any_sync(kFull, live)) {
            if (drained) break;
            continue;
        }
        w.round(tr, STEPS, stack, any_hit != 0);
        int slot = -1;
        bool doubtful = false;
        if (live && w.have && budgeted && w.tests > spill.budget) {
            const uint32_t e = atomicAdd(any_hit ? doubt.count : spill.count, 1u);
            if (any_hit) {
                doubtful = true;
                if (e < doubt.cap) doubt.list[e] = k;
                w.stop();
            } else if (e < spill.cap) {
                slot = (int)e;
                w.stop();
            } else {
                budgeted = false;  // list full: finish here
            }
        }
        if (live && !w.have) {
            if (doubtful) {
                hits[k].id = kDoubtMark;
            } else {
                store_hit(hits + k, w.hit());
                if (slot >= 0) spill_record(list, slot, kHeavyRay, k);
                if (leaves) leaves[k] = tr.compact ? 1u : w.b.leaf;
            }
            live = false;
        }
    }
}

__global__ void __launch_bounds__(kTraceThreads, 6) k_trace_doubt(TreeRef tr, const rt_ray* __restrict__ rays,
                                                               uint32_t num_rays, const uint32_t* __restrict__ starts,
                                                               rt_hit* __restrict__ hits, uint32_t* __restrict__ leaves,
                                                               Doubt doubt, Spill spill, uint32_t* __restrict__ list) {
    constexpr uint32_t kFull = 0xffffffffu;
    grid_dep_wait();
    const bool marked = *doubt.count > doubt.cap;
    const uint32_t n = marked ? num_rays : *doubt.count;
    const int lane = threadIdx.x & 31;
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    uint32_t k = 0;
    bool live = false, budgeted = spill.count != nullptr, drained = false;
    // few rays are spread over all warps, some lanes of each
    const uint32_t warps = gridDim.x * (kTraceThreads / 32), per = max(1u, (n + warps - 1) / warps);
    const uint32_t lanes = per < 32u ? (1u << per) - 1u : kFull;
    for (;;) {
        const uint32_t idle = __ballot_sync(kFull, !live) & lanes;
        if (!drained && (idle == lanes || __popc(idle) >= kRayRefill)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(doubt.work, (uint32_t)__popc(idle));
            base = __shfl_sync(kFull, base, 0);
            if (base >= n || n - base <= (uint32_t)__popc(idle)) drained = true;
            const uint32_t q = base + __popc(idle & ((1u << lane) - 1u));
            bool take = ((idle >> lane) & 1u) && base < n && q < n;
            if (take && marked) take = hits[q].id == kDoubtMark;
            if (take) {
                k = marked ? q : doubt.list[q];
                live = true;
            }
            w.start(take, load_ray(rays, k, take), tr, (starts && take) ? __ldg(starts + k) : 1u, stack, true);
        }
        if (!__any_sync(kFull, live)) {
            if (drained) break;
            continue;
        }
        const bool tested = w.round(tr, kRaySteps, stack, true);
        int slot = -1;
        if (live && tested && w.b.id < 0 && w.more && budgeted && w.at_leaf > spill.budget) {
            const uint32_t e = atomicAdd(spill.count, 1u);
            if (e < spill.cap) {
                slot = (int)e;
                w.stop();
            } else {
                budgeted = false;
            }
        }
        if (live && !w.have) {
            if (slot >= 0) {
                spill_record(list, slot, kHeavyRay, k);
            } else {
                store_hit(hits + k, w.hit());
                if (leaves) leaves[k] = tr.compact ? 1u : w.b.leaf;
            }
            live = false;
        }
    }
}

template <bool STATS>
__global__ void __launch_bounds__(kTraceThreads) k_trace_rays(TreeRef tr, const rt_ray* __restrict__ rays, uint32_t n,
                                                              int any_hit, const uint32_t* __restrict__ starts,
                                                              rt_hit* __restrict__ hits, uint32_t* __restrict__ leaves,
                                                              uint32_t* __restrict__ stats, uint32_t* work,
                                                              Spill spill, uint32_t* __restrict__ list,
                                                              TileOrder ord) {
    const uint32_t num_tiles = (n + 31) / 32;
    const uint32_t wbuf = *ord.parity, rbuf = wbuf ^ 1u, heavy = min(ord.counts[rbuf], ord.cap);
    for (uint32_t tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles); tile < num_tiles;
         tile = next_ordered_tile(work, ord, rbuf, heavy, num_tiles)) {
        const uint32_t k = tile * 32 + (threadIdx.x & 31);
        const bool valid = k < n;
        const RayState r = load_ray(rays, k, valid);
        const uint32_t start = (starts && valid) ? __ldg(starts + k) : 1u;
        uint32_t nb = 0, nt = 0, leaf = 1;
        int slot = -1;
        const Hit h = trace_ray<STATS>(r, valid, tr, any_hit != 0, &nb, &nt, &spill, &slot, start, &leaf);
        if (valid) {
            store_hit(hits + k, h);  // of a handed-over ray: the closest hit so far
            if (slot >= 0) spill_record(list, slot, kHeavyRay, k);
            if (leaves) leaves[k] = leaf;
            if (STATS) {
                stats[2 * k] = nb;
                stats[2 * k + 1] = nt;
            }
        }
        record_tile_cost(ord, wbuf, tile, nb + nt);
    }
}

// Second pass over the rays the first pass handed over: one ray per warp, rebuilt
// from its list entry exactly as the first pass made it, and its result written where
// the first pass would have written it.  A closest hit is the one that the first pass
// would have found (trace_ordered), so the budget, and which tests count towards it,
// change no hit.
struct HeavyArgs {
    TreeRef tr;
    const float* soup;
    rt_camera cam;
    float lx, ly, lz;
    const rt_hit* prim;   // primary hits (shadow / mirror entries)
    const uint32_t* prim_leaves;  // and their leaves, where the shading rays start (nullable: the root)
    rt_hit* hits;         // primary or generic-ray output
    uint8_t* vis;
    rt_hit* mirror;
    const rt_ray* rays;
    const uint32_t* starts;  // start nodes of generic rays (nullable)
    int any_hit;          // generic rays
    uint32_t* leaves;     // primary / generic-ray leaf output (nullable)
    uint32_t* mirror_leaves;
    uint32_t wide_cap;    // frontier-stack entries per warp (wide_stack_entries of the tree depth)
    uint32_t team_cap;    // frontier-stack entries per block (team_stack_entries of the tree depth)
    ShadeLists sl;        // primary entries: set up their pixel's shading rays too (sl.lists != nullptr)
    const uint32_t* list;
    const uint32_t* count;
    uint32_t cap;
    uint32_t* work;
    uint32_t* work2;      // claims of the block-per-ray pass
};

// The closest hit the first pass had found when it handed the ray over.
__device__ __forceinline__ Hit hit_so_far(const rt_hit* p) {
    const int4 v = __ldcg(reinterpret_cast<const int4*>(p));
    Hit h;
    h.id = v.x;
    h.u = __int_as_float(v.y);
    h.v = __int_as_float(v.z);
    h.t = __int_as_float(v.w);
    return h;
}
__device__ __forceinline__ Hit no_hit() {
    Hit h;
    h.id = -1;
    h.u = h.v = -1.0f;
    h.t = 0.0f;
    return h;
}

__device__ __forceinline__ bool heavy_any_hit(const HeavyArgs& a, uint32_t entry) {
    const uint32_t kind = entry >> 30;
    return kind == kHeavyShadow || (kind == kHeavyRay && a.any_hit);
}

__device__ __forceinline__ ShadeRays heavy_shade_rays(const HeavyArgs& a, uint32_t idx, bool mirror, uint32_t* start) {
    const uint32_t i = idx % a.cam.width, j = idx / a.cam.width;
    const int4 ph = __ldg(reinterpret_cast<const int4*>(a.prim + idx));
    *start = shade_start(a.prim_leaves, ph, true, idx);
    return shade_rays(a.soup, a.cam, a.lx, a.ly, a.lz, ph, true, i, j, mirror);
}

// A closest-hit entry, by a warp.
__device__ __forceinline__ void heavy_closest(const HeavyArgs& a, uint32_t entry) {
    const int lane = threadIdx.x & 31;
    const uint32_t kind = entry >> 30, idx = entry & kHeavyIndexMask;
    RayState r;
    uint32_t start = 1u;
    rt_hit* out = a.hits + idx;
    uint32_t* leaves = a.leaves;
    if (kind == kHeavyPrimary) {
        r = make_ray(mk3(a.cam.eye[0], a.cam.eye[1], a.cam.eye[2]), primary_dir(a.cam, idx % a.cam.width, idx / a.cam.width),
                     1e16f, -1);
    } else if (kind == kHeavyRay) {
        r = load_ray(a.rays, idx, true);
        if (a.starts) start = __ldg(a.starts + idx);
    } else {
        r = heavy_shade_rays(a, idx, true, &start).mirror;
        out = a.mirror + idx;
        leaves = a.mirror_leaves;
    }
    uint32_t leaf = 1u;
    const Hit h = trace_ordered(r, a.tr, a.wide_cap, hit_so_far(out), start, leaves ? &leaf : nullptr);
    if (leaves && leaf == 0u) leaf = __ldcg(leaves + idx);  // the first pass's
    __syncwarp();
    if (lane == 0) {
        store_hit(out, h);
        if (leaves) leaves[idx] = leaf;
    }
    if (kind == kHeavyPrimary && a.sl.lists) {
        const int4 ph = make_int4(h.id, __float_as_int(h.u), __float_as_int(h.v), __float_as_int(h.t));
        shade_setup_pixel(a.sl, a.cam, ph, lane == 0, idx % a.cam.width, idx / a.cam.width, idx, leaf);
    }
}

// ANY: the list holds a caller's any-hit rays alone (the ordered walk's registers would cost such
// calls a block per SM).
template <bool ANY>
__global__ void __launch_bounds__(kTraceThreads, ANY ? 7 : 6) k_trace_heavy(HeavyArgs a) {
    grid_dep_wait();
    const uint32_t n = min(*a.count, a.cap);
    const int lane = threadIdx.x & 31;
    for (uint32_t e = next_tile(a.work); e < n; e = next_tile(a.work)) {
        const uint32_t entry = __ldg(a.list + e);
        const uint32_t idx = entry & kHeavyIndexMask;
        if (!ANY && !heavy_any_hit(a, entry)) {
            heavy_closest(a, entry);
        } else if (ANY || (entry >> 30) == kHeavyRay) {
            const Hit h = trace_wide(load_ray(a.rays, idx, true), a.tr, a.wide_cap);
            if (lane == 0) {
                store_hit(a.hits + idx, h);
                if (a.leaves) a.leaves[idx] = 1u;
            }
        } else {
            uint32_t start;
            const ShadeRays s = heavy_shade_rays(a, idx, false, &start);
            const Hit h = trace_wide(s.shadow, a.tr, a.wide_cap);
            if (lane == 0) a.vis[idx] = vis_code(s.has, s.cast, h.id >= 0);
        }
    }
}

// A few closest-hit rays, a warp each from the start: with a lane each they fill
// a handful of warps, and the call lasts as long as the longest chain of dependent
// loads.  256 rays over 65 k triangles 66 -> 19 us; 16,384 rays at a torus of 65 k triangles, at
// 260 k and in a soup of 200 k 109, 112 and 114 us (lanes 163, 157 and 173), 24,000 152,
// 158 and 161 (165, 158 and 180).  Rays along an axis of a mesh are the exception: 18,000 over 260 k
// triangles 116 us, with lanes 82.
constexpr uint32_t kFewRays = 16384;

__global__ void __launch_bounds__(kTraceThreads) k_rays_wide(TreeRef tr, const rt_ray* __restrict__ rays, uint32_t n,
                                                             const uint32_t* __restrict__ starts,
                                                             rt_hit* __restrict__ hits, uint32_t cap) {
    grid_dep_wait();
    const uint32_t k = blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (k >= n) return;
    const Hit h = trace_ordered(load_ray(rays, k, true), tr, cap, no_hit(), starts ? __ldg(starts + k) : 1u, nullptr);
    if ((threadIdx.x & 31) == 0) store_hit(hits + k, h);
}

// k_trace_heavy with a block per any-hit ray (traverse_team): for the handed-over
// shading rays, a few hundred grazing rays whose walks run for thousands of
// tests, where a warp per ray leaves the GPU waiting on the longest few.  The closest-hit
// entries come first, a warp each (a block each: 3 us of 1,400 for the mirror rays of
// 2.1 M triangles at 1080p).
__global__ void __launch_bounds__(kTeamThreads, 6) k_trace_heavy_team(HeavyArgs a) {
    grid_dep_wait();
    __shared__ TeamShared ts;
    __shared__ uint32_t s_e;
    const uint32_t n = min(*a.count, a.cap);
    const int tid = threadIdx.x;
    for (uint32_t e = next_tile(a.work); e < n; e = next_tile(a.work)) {
        const uint32_t entry = __ldg(a.list + e);
        if (!heavy_any_hit(a, entry)) heavy_closest(a, entry);
    }
    for (;;) {
        __syncthreads();
        if (tid == 0) s_e = atomicAdd(a.work2, 1u);
        __syncthreads();
        const uint32_t e = s_e;
        if (e >= n) break;
        const uint32_t entry = __ldg(a.list + e);
        const uint32_t idx = entry & kHeavyIndexMask;
        if (!heavy_any_hit(a, entry)) continue;
        if ((entry >> 30) == kHeavyRay) {
            const Hit h = trace_team(load_ray(a.rays, idx, true), a.tr, a.team_cap, ts);
            if (tid == 0) {
                store_hit(a.hits + idx, h);
                if (a.leaves) a.leaves[idx] = 1u;
            }
        } else {
            uint32_t start;
            const ShadeRays s = heavy_shade_rays(a, idx, false, &start);
            const Hit h = trace_team(s.shadow, a.tr, a.team_cap, ts);
            if (tid == 0) a.vis[idx] = vis_code(s.has, s.cast, h.id >= 0);
        }
    }
}

uint32_t pixel_tiles(const rt_camera* cam) {
    return (uint32_t)(((cam->width + 7) / 8) * ((cam->height + 3) / 4));
}

rt_status check_trace_args(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, const char* who) {
    if (!ctx) return RT_ERR_INVALID;
    if (!l || !cam) return rt_fail(ctx, RT_ERR_INVALID, "%s: null argument", who);
    if (l->n == 0) return rt_fail(ctx, RT_ERR_INVALID, "%s: the LBVH has not been built", who);
    if (cam->width == 0 || cam->height == 0 || (uint64_t)cam->width * cam->height > (1ull << 31))
        return rt_fail(ctx, RT_ERR_INVALID, "%s: bad image size %ux%u", who, cam->width, cam->height);
    return RT_OK;
}

}  // namespace

rt_status ensure_shade_lists(rt_ctx* ctx, rt_lbvh* l, size_t px) {
    if (px <= l->s_pixels) return RT_OK;
    if (l->graph_refs > 0)
        return rt_fail(ctx, RT_ERR_CAPACITY,
                       "shading lists of %zu pixels cannot grow to %zu while a captured frame uses them",
                       l->s_pixels, px);
    RT_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (l->s_lists) cudaFree(l->s_lists);
    if (l->s_rays) cudaFree(l->s_rays);
    l->s_lists = nullptr;
    l->s_rays = nullptr;
    l->s_pixels = 0;
    // shadow-ray pixels, mirror-ray pixels, primary leaves of a frame, start
    // nodes of the listed rays (2 x px); the listed rays (2 x px x 32 bytes)
    RT_CHECK_CUDA(ctx, cudaMalloc((void**)&l->s_lists, 5 * sizeof(uint32_t) * px));
    RT_CHECK_CUDA(ctx, cudaMalloc((void**)&l->s_rays, 4 * sizeof(float4) * px));
    l->s_pixels = px;
    return RT_OK;
}

TreeRef tree_ref(const rt_ctx* ctx, const rt_lbvh* l) {
    TreeRef t;
    t.compact = l->compact_valid;
    t.tri_base = 0;
    t.nodes = t.compact ? l->cnodes : l->nodes;
    t.num_nodes = t.compact ? l->ccap : l->num_nodes;
    t.tris = l->sorted_tris;
    t.n = l->n;
    t.err = ctx->d_err;
    t.heap = l->nodes;
    t.num_heap = l->num_nodes;
    t.tnodes = l->tnodes;
    t.leaf_of = l->leaf_of;
    t.num_tnodes = l->num_nodes / 2;
    t.records_valid = l->counters + 7;
    return t;
}

namespace {

// Heavy-ray hand-over of one trace call: the list is emptied before the
// first pass (budget 0 or a counting pass: no hand-over), and the second pass
// drains it.
// The shading rays keep their own list length and claim counter, so a frame
// zeroes both passes' counters in one launch before its primary pass.
Spill spill_of(rt_ctx* ctx, bool enabled, int kind) {
    Spill sp;
    sp.budget = ctx->trace_budget[kind];
    const bool shade = kind == 1;
    sp.count = (enabled && sp.budget) ? ctx->d_spill_count + (shade ? 1 : 0) : nullptr;
    sp.work = shade ? ctx->d_spill_count + 2 : ctx->d_work + kWorkHeavy;
    sp.cap = kSpillCap;
    return sp;
}

// Claims of the block-per-ray pass, one word for the shading rays and one for the others.
uint32_t* team_claims(const rt_ctx* ctx, const Spill& sp) {
    return ctx->d_words + kTeamClaims + (sp.work == ctx->d_spill_count + 2 ? 1 : 0);
}

// A trace call zeroes its counters (words of ctx->d_words) in one small
// kernel launched before its first pass, k_order_begin where the call has a
// tile order to advance, k_reset_words otherwise: one graph node instead of a
// memset per counter, and a programmatic edge to the pass.
uint64_t word_bit(const rt_ctx* ctx, const uint32_t* p) { return 1ull << (uint32_t)(p - ctx->d_words); }

// The list length and the second pass's claim counters.
uint64_t spill_reset_bits(const rt_ctx* ctx, const Spill& sp) {
    return sp.count ? word_bit(ctx, sp.count) | word_bit(ctx, sp.work) | word_bit(ctx, team_claims(ctx, sp)) : 0ull;
}

// The counters of the compacted shading-ray pass.
uint64_t shade_reset_bits(const rt_ctx* ctx, const Spill& sp) {
    return word_bit(ctx, ctx->d_work + kWorkSecondary) | word_bit(ctx, ctx->d_work + kWorkShade) |
           spill_reset_bits(ctx, sp);
}

__device__ __forceinline__ void zero_words(uint32_t* words, unsigned long long mask) {
    if (threadIdx.x < 64 && ((mask >> threadIdx.x) & 1ull)) words[threadIdx.x] = 0u;
}

Records no_records() {
    Records rec;
    memset(&rec, 0, sizeof(rec));
    return rec;
}

// Blocks past the first make the trace records of a tile each.
__global__ void __launch_bounds__(256) k_reset_words(uint32_t* words, unsigned long long mask, Records rec) {
    grid_dep_wait();
    if (blockIdx.x > 0) {
        make_records(rec, blockIdx.x - 1u);
        return;
    }
    zero_words(words, mask);
}

rt_status reset_words(rt_ctx* ctx, uint64_t mask, const Records& rec) {
    if (!mask && !rec.tiles) return RT_OK;
    launch_pdl(k_reset_words, 1u + rec.tiles * rec.slices, rec.tiles ? 256 : 64, 0, ctx->stream, ctx->d_words, (unsigned long long)mask,
               rec);
    RT_CHECK_LAUNCH(ctx, "k_reset_words");
    return RT_OK;
}

rt_status launch_heavy(rt_ctx* ctx, const Spill& sp, HeavyArgs a, int kind) {
    if (!sp.count) return RT_OK;
    a.list = ctx->d_spill;
    a.count = sp.count;
    a.cap = kSpillCap;
    a.work = sp.work;
    a.work2 = team_claims(ctx, sp);
    if ((ctx->heavy_team >> kind) & 1u) {
        const size_t smem = std::max(team_smem_bytes(a.team_cap), wide_smem_bytes(a.wide_cap));
        if (smem > 48u * 1024u)
            RT_CHECK_CUDA(ctx, cudaFuncSetAttribute(k_trace_heavy_team, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    (int)smem));
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trace_heavy_team, kTeamThreads, smem) !=
                cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        launch_pdl(k_trace_heavy_team, (uint32_t)per_sm * ctx->num_sms, kTeamThreads, smem, ctx->stream, a);
        RT_CHECK_LAUNCH(ctx, "k_trace_heavy_team");
        return RT_OK;
    }
    const size_t smem = wide_smem_bytes(a.wide_cap);
    const auto k = kind == 2 && a.any_hit ? k_trace_heavy<true> : k_trace_heavy<false>;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kTraceThreads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    launch_pdl(k, (uint32_t)per_sm * ctx->num_sms, kTraceThreads, smem, ctx->stream, a);
    RT_CHECK_LAUNCH(ctx, "k_trace_heavy");
    return RT_OK;
}

__global__ void __launch_bounds__(256) k_order_begin(TileOrder o, uint32_t* words, unsigned long long reset, Records rec) {
    grid_dep_wait();
    if (blockIdx.x > 0) {
        make_records(rec, blockIdx.x - 1u);
        return;
    }
    zero_words(words, reset);
    __shared__ uint32_t s_w;
    if (threadIdx.x == 0) {
        const uint32_t w = *o.parity ^ 1u;
        *o.parity = w;
        s_w = w;
    }
    __syncthreads();
    const uint32_t w = s_w;
    const uint32_t n = min(o.counts[w], o.cap);
    __syncthreads();
    // the buffer this call writes was read two calls ago: clear its bits
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        const uint32_t t = o.lists[(size_t)w * o.cap + i];
        if (t < o.cap) o.bits[(size_t)w * (o.cap / 32) + t / 32] = 0u;
    }
    __syncthreads();
    if (threadIdx.x == 0) o.counts[w] = 0u;
}

// Tile order of one trace kind (0 primary, 1 shading, 2 generic rays),
// advanced to this call; enabled == false gives image order (cap 0: no list
// is read or written).  reset: the call's counters to zero (word_bit mask).
// l (nullable): the tree whose trace records the call needs.
rt_status order_begin(rt_ctx* ctx, int kind, bool enabled, TileOrder* out, uint64_t reset = 0,
                      const rt_lbvh* l = nullptr) {
    TileOrder o;
    o.cap = enabled ? kOrderCap : 0u;
    o.parity = ctx->d_words + 40 + 4 * kind;
    o.counts = o.parity + 1;
    o.lists = ctx->d_order + (size_t)kind * kOrderWords;
    o.bits = o.lists + 2 * (size_t)kOrderCap;
    if (enabled) {
        const Records rec = l ? records_of(ctx, l) : no_records();
        launch_pdl(k_order_begin, 1u + rec.tiles * rec.slices, 256, 0, ctx->stream, o, ctx->d_words, (unsigned long long)reset, rec);
        RT_CHECK_LAUNCH(ctx, "k_order_begin");
    } else {
        rt_status s = reset_words(ctx, reset, l ? records_of(ctx, l) : no_records());
        if (s != RT_OK) return s;
    }
    *out = o;
    return RT_OK;
}

HeavyArgs heavy_args(rt_ctx* ctx, const rt_lbvh* l) {
    HeavyArgs a;
    memset(&a, 0, sizeof(a));
    a.tr = tree_ref(ctx, l);
    a.wide_cap = wide_stack_entries(l->depth);
    a.team_cap = team_stack_entries(l->depth);
    return a;
}

}  // namespace

namespace {

// sl (nullable): a frame's shading lists, filled by this pass as it goes
// (their counts are zeroed with this call's counters); the statistics
// variant never fills them.
rt_status trace_primary(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, rt_hit* d_hits, uint32_t* d_leaves,
                        uint32_t* d_stats, const char* who, const ShadeLists* sl = nullptr,
                        uint64_t extra_reset = 0) {
    rt_status s = check_trace_args(ctx, l, cam, who);
    if (s != RT_OK) return s;
    if (!d_hits) return rt_fail(ctx, RT_ERR_INVALID, "%s: null output", who);
    const Spill sp = spill_of(ctx, !d_stats && (uint64_t)cam->width * cam->height <= kHeavyIndexMask, 0);
    uint64_t reset = word_bit(ctx, ctx->d_work + kWorkPrimary) | spill_reset_bits(ctx, sp) | extra_reset;
    if (sl && !d_stats) reset |= word_bit(ctx, sl->counts) | word_bit(ctx, sl->counts + 1);
    TileOrder ord;
    if ((s = order_begin(ctx, 0, ctx->tile_order & 1u, &ord, reset, d_stats ? nullptr : l)) != RT_OK) return s;
    const uint32_t tiles = pixel_tiles(cam);
    uint32_t* work = ctx->d_work + kWorkPrimary;
    ShadeLists none;
    memset(&none, 0, sizeof(none));
    const ShadeLists lists = (sl && !d_stats) ? *sl : none;
    if (d_stats) {
        k_trace_primary<<<persistent_blocks(ctx, k_trace_primary, kTraceThreads, tiles), kTraceThreads, 0,
                          ctx->stream>>>(tree_ref(ctx, l), *cam, d_hits, d_leaves, d_stats, work, tiles, ord);
    } else {
        auto k = prim_blocks(ctx, tiles) == 8u ? k_walk_primary<8> : k_walk_primary<7>;
        launch_pdl(k, persistent_blocks(ctx, k, kTraceThreads, tiles), kTraceThreads, 0, ctx->stream, tree_ref(ctx, l), *cam, d_hits, d_leaves, work, tiles, sp, ctx->d_spill, ord, lists);
    }
    RT_CHECK_LAUNCH(ctx, d_stats ? "k_trace_primary" : "k_walk_primary");
    HeavyArgs a = heavy_args(ctx, l);
    a.cam = *cam;
    a.hits = d_hits;
    a.leaves = d_leaves;
    a.sl = lists;
    return launch_heavy(ctx, sp, a, 0);
}

// prebuilt: the frame's primary pass has filled the shading lists (and the
// results that need no ray), so the setup pass is skipped, and the counters
// of this pass were zeroed with the primary pass's (shade_reset_bits).
rt_status trace_shadow_mirror(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, const float light[3],
                              const rt_hit* d_primary, const uint32_t* d_prim_leaves, uint8_t* d_vis,
                              rt_hit* d_mirror, uint32_t* d_mirror_leaves, uint32_t* d_shadow_stats,
                              uint32_t* d_mirror_stats, const char* who, bool prebuilt = false) {
    rt_status s = check_trace_args(ctx, l, cam, who);
    if (s != RT_OK) return s;
    if (!light || !d_primary) return rt_fail(ctx, RT_ERR_INVALID, "%s: null argument", who);
    if (!l->src_tris) return rt_fail(ctx, RT_ERR_INVALID, "%s: no triangle soup bound", who);
    const bool stats = d_shadow_stats || d_mirror_stats;
    const Spill sp = spill_of(ctx, !stats && (uint64_t)cam->width * cam->height <= kHeavyIndexMask, 1);
    uint64_t reset = word_bit(ctx, ctx->d_work + kWorkSecondary) | spill_reset_bits(ctx, sp);
    const uint32_t tiles = pixel_tiles(cam);
    if (stats) {  // per-pixel counts in the oracle's order: the tile pass
        TileOrder ord;
        if ((s = order_begin(ctx, 1, ctx->tile_order & 2u, &ord, reset)) != RT_OK) return s;
        uint32_t* work = ctx->d_work + kWorkSecondary;
        k_trace_secondary<<<persistent_blocks(ctx, k_trace_secondary, kTraceThreads, tiles), kTraceThreads, 0,
                            ctx->stream>>>(tree_ref(ctx, l), l->src_tris, *cam, light[0], light[1], light[2], d_primary,
                                           d_prim_leaves, d_vis, d_mirror, d_mirror_leaves, d_shadow_stats,
                                           d_mirror_stats, work, tiles, ord);
        RT_CHECK_LAUNCH(ctx, "k_trace_secondary");
    } else {  // compacted shading-ray lists
        const size_t px = (size_t)cam->width * cam->height;
        if ((s = ensure_shade_lists(ctx, const_cast<rt_lbvh*>(l), px)) != RT_OK) return s;
        uint32_t* counts = ctx->d_work + kShadeCounts;
        if (!prebuilt) {
            reset = shade_reset_bits(ctx, sp) | word_bit(ctx, counts) | word_bit(ctx, counts + 1);
            if ((s = reset_words(ctx, reset, records_of(ctx, l))) != RT_OK) return s;
        }
        const uint32_t cap = (uint32_t)l->s_pixels;
        if (!prebuilt) {
            const uint32_t sblocks = std::max(1u, std::min((tiles + 7) / 8, (uint32_t)ctx->num_sms * 8));
            k_shade_setup<<<sblocks, 256, 0, ctx->stream>>>(l->src_tris, *cam, light[0], light[1], light[2], d_primary,
                                                             d_vis, d_mirror, d_mirror_leaves, d_prim_leaves,
                                                             l->s_lists, cap, counts, l->s_rays,
                                                             l->s_lists + 3 * l->s_pixels,
                                                             tiles);
            RT_CHECK_LAUNCH(ctx, "k_shade_setup");
        }
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_walk_shade<false>, kTraceThreads, 0) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
        launch_pdl(k_walk_shade<false>, (uint32_t)per_sm * ctx->num_sms, kTraceThreads, 0, ctx->stream, tree_ref(ctx, l), d_vis,
                   d_mirror, d_mirror_leaves, (const uint32_t*)l->s_lists, cap, (const uint32_t*)counts,
                   (const float4*)l->s_rays, (const uint32_t*)(l->s_lists + 3 * l->s_pixels), ctx->d_work + kWorkShade,
                   sp, ctx->d_spill, BatchTrees{nullptr, nullptr, nullptr, 0u, 0u});
        RT_CHECK_LAUNCH(ctx, "k_walk_shade");
    }
    HeavyArgs a = heavy_args(ctx, l);
    a.soup = l->src_tris;
    a.cam = *cam;
    a.lx = light[0];
    a.ly = light[1];
    a.lz = light[2];
    a.prim = d_primary;
    a.prim_leaves = d_prim_leaves;
    a.vis = d_vis;
    a.mirror = d_mirror;
    a.mirror_leaves = d_mirror_leaves;
    return launch_heavy(ctx, sp, a, 1);
}

rt_status trace_rays(rt_ctx* ctx, const rt_lbvh* l, const rt_ray* d_rays, uint32_t n, int any_hit,
                     const uint32_t* d_starts, rt_hit* d_hits, uint32_t* d_leaves, uint32_t* d_stats,
                     const char* who) {
    if (!ctx) return RT_ERR_INVALID;
    if (!l || !d_rays || !d_hits) return rt_fail(ctx, RT_ERR_INVALID, "%s: null argument", who);
    if (l->n == 0) return rt_fail(ctx, RT_ERR_INVALID, "%s: the LBVH has not been built", who);
    if (n == 0) return RT_OK;
    const Spill sp = spill_of(ctx, !d_stats && n <= kHeavyIndexMask, 2);
    const uint64_t reset = word_bit(ctx, ctx->d_work + kWorkRays) | spill_reset_bits(ctx, sp) |
                           word_bit(ctx, ctx->d_words + kDoubtCount) | word_bit(ctx, ctx->d_words + kDoubtCount + 1);
    TileOrder ord;
    if (!d_stats && !any_hit && !d_leaves && n <= kFewRays) {
        const uint32_t cap = wide_stack_entries(l->depth);
        launch_pdl(k_rays_wide, (n + kWideWarps - 1) / kWideWarps, kTraceThreads, wide_smem_bytes(cap), ctx->stream,
                   tree_ref(ctx, l), d_rays, n, d_starts, d_hits, cap);
        RT_CHECK_LAUNCH(ctx, "k_rays_wide");
        return RT_OK;
    }
    const bool walk = !d_stats && !(ctx->tile_order & 4u) && !(any_hit && (n < kWalkAnyRays || d_starts));
    rt_status s = order_begin(ctx, 2, ctx->tile_order & 4u, &ord, reset, walk ? l : nullptr);
    if (s != RT_OK) return s;
    const uint32_t tiles = (n + 31) / 32;
    uint32_t* work = ctx->d_work + kWorkRays;
    if (d_stats) {
        auto k = k_trace_rays<true>;
        k<<<persistent_blocks(ctx, k, kTraceThreads, tiles), kTraceThreads, 0, ctx->stream>>>(
            tree_ref(ctx, l), d_rays, n, any_hit, d_starts, d_hits, d_leaves, d_stats, work, sp, ctx->d_spill, ord);
    } else if (walk) {
        const Doubt doubt{ctx->d_spill + kSpillCap, ctx->d_words + kDoubtCount, ctx->d_words + kDoubtCount + 1,
                          ctx->doubt_limit};
        auto k = n <= ray_lanes(ctx) ? k_walk_rays<kFewSteps> : k_walk_rays<kRaySteps>;
        launch_pdl(k, persistent_blocks(ctx, k, kTraceThreads, tiles), kTraceThreads, 0, ctx->stream,
                   tree_ref(ctx, l), d_rays, n, any_hit, d_starts, d_hits, d_leaves, work, sp, ctx->d_spill, doubt);
        if (any_hit && sp.count) {
            RT_CHECK_LAUNCH(ctx, "k_walk_rays");
            launch_pdl(k_trace_doubt, persistent_blocks(ctx, k_trace_doubt, kTraceThreads, tiles), kTraceThreads, 0,
                       ctx->stream, tree_ref(ctx, l), d_rays, n, d_starts, d_hits, d_leaves, doubt, sp, ctx->d_spill);
        }
    } else {
        auto k = k_trace_rays<false>;
        k<<<persistent_blocks(ctx, k, kTraceThreads, tiles), kTraceThreads, 0, ctx->stream>>>(
            tree_ref(ctx, l), d_rays, n, any_hit, d_starts, d_hits, d_leaves, nullptr, work, sp, ctx->d_spill, ord);
    }
    RT_CHECK_LAUNCH(ctx, walk ? (any_hit ? "k_trace_doubt" : "k_walk_rays") : "k_trace_rays");
    HeavyArgs a = heavy_args(ctx, l);
    a.rays = d_rays;
    a.starts = d_starts;
    a.any_hit = any_hit;
    a.hits = d_hits;
    a.leaves = d_leaves;
    return launch_heavy(ctx, sp, a, 2);
}

}  // namespace

Spill shadow_spill(rt_ctx* ctx) { return spill_of(ctx, true, 1); }

// Zeroes the counters of a bounce of the colour stage (words of ctx->d_words and the
// shadow rays' hand-over) and makes the trace records if the tree has none.
rt_status begin_bounce(rt_ctx* ctx, const rt_lbvh* l, const Spill& shadow, std::initializer_list<uint32_t*> words) {
    uint64_t mask = spill_reset_bits(ctx, shadow);
    for (uint32_t* w : words) mask |= word_bit(ctx, w);
    return reset_words(ctx, mask, records_of(ctx, l));
}

rt_status reset_work_and_records(rt_ctx* ctx, int slot, const rt_lbvh* l, uint64_t words) {
    return reset_words(ctx, words | word_bit(ctx, ctx->d_work + slot), records_of(ctx, l));
}

extern "C" rt_status rt_trace_primary(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, rt_hit* d_hits,
                                      uint32_t* d_stats) {
    return trace_primary(ctx, l, cam, d_hits, nullptr, d_stats, "rt_trace_primary");
}

extern "C" rt_status rt_trace_primary_leaves(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, rt_hit* d_hits,
                                             uint32_t* d_leaves, uint32_t* d_stats) {
    return trace_primary(ctx, l, cam, d_hits, d_leaves, d_stats, "rt_trace_primary_leaves");
}

extern "C" rt_status rt_trace_shadow_mirror(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam, const float light[3],
                                            const rt_hit* d_primary, uint8_t* d_vis, rt_hit* d_mirror,
                                            uint32_t* d_shadow_stats, uint32_t* d_mirror_stats) {
    return trace_shadow_mirror(ctx, l, cam, light, d_primary, nullptr, d_vis, d_mirror, nullptr, d_shadow_stats,
                               d_mirror_stats, "rt_trace_shadow_mirror");
}

extern "C" rt_status rt_trace_shadow_mirror_from(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam,
                                                 const float light[3], const rt_hit* d_primary,
                                                 const uint32_t* d_primary_leaves, uint8_t* d_vis, rt_hit* d_mirror,
                                                 uint32_t* d_mirror_leaves, uint32_t* d_shadow_stats,
                                                 uint32_t* d_mirror_stats) {
    return trace_shadow_mirror(ctx, l, cam, light, d_primary, d_primary_leaves, d_vis, d_mirror, d_mirror_leaves,
                               d_shadow_stats, d_mirror_stats, "rt_trace_shadow_mirror_from");
}

extern "C" rt_status rt_trace_rays(rt_ctx* ctx, const rt_lbvh* l, const rt_ray* d_rays, uint32_t n, int any_hit,
                                   rt_hit* d_hits, uint32_t* d_stats) {
    return trace_rays(ctx, l, d_rays, n, any_hit, nullptr, d_hits, nullptr, d_stats, "rt_trace_rays");
}

extern "C" rt_status rt_trace_rays_from(rt_ctx* ctx, const rt_lbvh* l, const rt_ray* d_rays, uint32_t n, int any_hit,
                                        const uint32_t* d_starts, rt_hit* d_hits, uint32_t* d_leaves,
                                        uint32_t* d_stats) {
    return trace_rays(ctx, l, d_rays, n, any_hit, d_starts, d_hits, d_leaves, d_stats, "rt_trace_rays_from");
}

// The trace stages of one frame: primary rays, then the shading rays started
// at each primary hit's leaf (the iRoot restart; the leaves live in the third
// segment of the shading lists, which the caller has sized).
rt_status trace_frame(rt_ctx* ctx, rt_lbvh* l, const rt_camera* cam, const float light[3], rt_hit* d_primary,
                      uint8_t* d_vis, rt_hit* d_mirror, const char* who) {
    const size_t px = (size_t)cam->width * cam->height;
    uint32_t* leaves = (d_vis || d_mirror) && l->s_pixels >= px ? l->s_lists + 2 * l->s_pixels : nullptr;
    if (!leaves) return trace_primary(ctx, l, cam, d_primary, nullptr, nullptr, who);
    if (!l->src_tris) return rt_fail(ctx, RT_ERR_INVALID, "%s: no triangle soup bound", who);
    // the primary pass (and its warp-per-ray pass) fills the shading lists
    ShadeLists sl{l->src_tris, light[0], light[1], light[2], d_vis,     d_mirror,
                  l->s_lists, (uint32_t)l->s_pixels, ctx->d_work + kShadeCounts, l->s_rays,
                  l->s_lists + 3 * l->s_pixels};
    // the shading pass's counters are zeroed with the primary pass's
    const Spill ssp = spill_of(ctx, px <= kHeavyIndexMask, 1);
    rt_status s = trace_primary(ctx, l, cam, d_primary, leaves, nullptr, who, &sl, shade_reset_bits(ctx, ssp));
    if (s == RT_OK)
        s = trace_shadow_mirror(ctx, l, cam, light, d_primary, leaves, d_vis, d_mirror, nullptr, nullptr, nullptr, who,
                                true);
    return s;
}

rt_status ensure_frame_buffers(rt_ctx* ctx, rt_lbvh* l, size_t px) {
    if (px <= l->f_pixels) return RT_OK;  // frame buffers grow on the first call at a new size
    if (l->graph_refs > 0)
        return rt_fail(ctx, RT_ERR_CAPACITY,
                       "frame buffers of %zu pixels cannot grow to %zu while a captured frame uses them",
                       l->f_pixels, px);
    RT_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (l->f_primary) cudaFree(l->f_primary);
    if (l->f_mirror) cudaFree(l->f_mirror);
    if (l->f_vis) cudaFree(l->f_vis);
    l->f_primary = nullptr; l->f_mirror = nullptr; l->f_vis = nullptr; l->f_pixels = 0;
    RT_CHECK_CUDA(ctx, cudaMalloc((void**)&l->f_primary, sizeof(rt_hit) * px));
    RT_CHECK_CUDA(ctx, cudaMalloc((void**)&l->f_mirror, sizeof(rt_hit) * px));
    RT_CHECK_CUDA(ctx, cudaMalloc((void**)&l->f_vis, px));
    l->f_pixels = px;
    return RT_OK;
}

static rt_status render_frame_host(rt_ctx* ctx, rt_lbvh* l, const float* h_tris, uint32_t n, const rt_camera* cam,
                                   const float light[3], rt_hit* h_primary, uint8_t* h_vis, rt_hit* h_mirror,
                                   bool sync, const char* who) {
    if (!ctx) return RT_ERR_INVALID;
    if (!l || !h_tris || !cam || !light) return rt_fail(ctx, RT_ERR_INVALID, "%s: null argument", who);
    const size_t px = (size_t)cam->width * cam->height;
    if (px == 0 || px > (1ull << 31)) return rt_fail(ctx, RT_ERR_INVALID, "%s: bad image size", who);
    rt_status s = ensure_frame_buffers(ctx, l, px);
    if (s != RT_OK) return s;
    if (h_vis || h_mirror) {
        if ((s = ensure_shade_lists(ctx, l, px)) != RT_OK) return s;
    }
    if ((s = rt_lbvh_build_host(ctx, l, h_tris, n, 0)) != RT_OK) return s;
    if ((s = trace_frame(ctx, l, cam, light, l->f_primary, h_vis ? l->f_vis : nullptr, h_mirror ? l->f_mirror : nullptr,
                         who)) != RT_OK)
        return s;
    cudaStream_t st = ctx->stream;
    if (h_primary) RT_CHECK_CUDA(ctx, cudaMemcpyAsync(h_primary, l->f_primary, sizeof(rt_hit) * px, cudaMemcpyDeviceToHost, st));
    if (h_vis) RT_CHECK_CUDA(ctx, cudaMemcpyAsync(h_vis, l->f_vis, px, cudaMemcpyDeviceToHost, st));
    if (h_mirror) RT_CHECK_CUDA(ctx, cudaMemcpyAsync(h_mirror, l->f_mirror, sizeof(rt_hit) * px, cudaMemcpyDeviceToHost, st));
    if (sync) RT_CHECK_CUDA(ctx, cudaStreamSynchronize(st));
    return RT_OK;
}

extern "C" rt_status rt_render_frame_host(rt_ctx* ctx, rt_lbvh* l, const float* h_tris, uint32_t n,
                                          const rt_camera* cam, const float light[3], rt_hit* h_primary,
                                          uint8_t* h_vis, rt_hit* h_mirror) {
    return render_frame_host(ctx, l, h_tris, n, cam, light, h_primary, h_vis, h_mirror, true, "rt_render_frame_host");
}

extern "C" rt_status rt_render_frame_host_async(rt_ctx* ctx, rt_lbvh* l, const float* h_tris, uint32_t n,
                                                const rt_camera* cam, const float light[3], rt_hit* h_primary,
                                                uint8_t* h_vis, rt_hit* h_mirror) {
    return render_frame_host(ctx, l, h_tris, n, cam, light, h_primary, h_vis, h_mirror, false,
                             "rt_render_frame_host_async");
}

// ---------------------------------------------------------------------------
// The frame in the reference's own walk order: LBVH_IntersectP
// (LBVH.hlsl:363-440) as the shader runs it, a stackless walk over the heap
// driven by a trail word, one box test per visited node, the child picked by
// dirIsNeg[axis field] first, leaf triangles tested in order and a
// candidate kept only when strictly nearer (an exact tie keeps the first
// one tested, as the shader does).  Primary rays start at the root; the
// shadow ray (a closest-hit walk, as CSComputeColorRT.hlsl:160 issues it)
// and the mirror ray restart at the primary hit's leaf (iRoot).  One lane
// per ray.  Its per-ray counts are the shader's iVisitedNodes (visited nodes,
// triangle tests), the figures the trace's algorithmic bytes are defined by.
namespace {

template <bool EXACT>
__device__ __forceinline__ Hit shader_walk(const RayState& r, bool active, const TreeRef& tr, uint32_t node,
                                           uint32_t* visits_out, uint32_t* ntri_out, uint32_t* leaf_out) {
    Hit best;
    best.id = -1;
    best.u = -1.0f;
    best.v = -1.0f;
    best.t = r.tmax;
    uint32_t root = 1, visits = 0, ntri = 0;
    if (node < 1u) node = 1u;
    uint32_t trail = 1u << (31 - __clz(node));
    const uint32_t limit = 2u * tr.num_nodes + 64u;  // a tree walk visits each node once at most
    while (active) {
        if (node >= tr.num_nodes || visits >= limit) {
            atomicOr(tr.err, RT_DEVERR_BOUNDS);
            break;
        }
        const NodeBox nb = load_node(tr.nodes, node);
        const int p = __ffs(trail + 1u) - 1;
        ++visits;
        float t0;
        // IntersectBox, entered unless T0 > closest t or T1 < 0
        if (!box_enter<EXACT>(r, nb.a.x, nb.a.y, nb.a.z, nb.a.w, nb.b.x, nb.b.y, best.t, &t0)) {
            trail = (trail >> p) + 1u;
            node = (node >> p) ^ 1u;
        } else if (__float_as_int(nb.b.z) & 4) {
            const int cnt = __float_as_int(nb.b.z) >> 3, pos = __float_as_int(nb.b.w);
            if (pos < 0 || cnt < 0 || (uint32_t)pos + (uint32_t)cnt > tr.n) {
                atomicOr(tr.err, RT_DEVERR_BOUNDS);
                break;
            }
            for (int i = 0; i < cnt; ++i) {
                const float4* tp = tr.tris + 3 * (size_t)(pos + i);
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                ++ntri;
                const int id = __float_as_int(a.w);
                float u, v, t;
                if (id != r.exclude && tri_test(r, a, b, c, &u, &v, &t) && t < best.t) {
                    best.id = id;
                    best.u = u;
                    best.v = v;
                    best.t = t;
                    root = node;
                }
            }
            trail = (trail >> p) + 1u;
            node = (node >> p) ^ 1u;
        } else {
            const int field = __float_as_int(nb.b.z) & 3;
            const float ia = field == 0 ? r.inv.x : (field == 1 ? r.inv.y : r.inv.z);
            trail <<= 1;
            node = (node << 1) | (ia < 0.0f ? 1u : 0u);
        }
        if (trail <= 1u) break;
    }
    if (visits_out) *visits_out = visits;
    if (ntri_out) *ntri_out = ntri;
    if (leaf_out) *leaf_out = root;
    return best;
}

__device__ __forceinline__ Hit shader_trace(const RayState& r, bool active, const TreeRef& tr, uint32_t node,
                                            uint32_t* visits, uint32_t* ntri, uint32_t* leaf) {
    if (__any_sync(0xffffffffu, active && r.exact)) return shader_walk<true>(r, active, tr, node, visits, ntri, leaf);
    return shader_walk<false>(r, active, tr, node, visits, ntri, leaf);
}

__global__ void __launch_bounds__(kTraceThreads) k_shader_primary(TreeRef tr, rt_camera cam, rt_hit* __restrict__ hits,
                                                                  uint32_t* __restrict__ leaves,
                                                                  uint32_t* __restrict__ stats, uint32_t* work,
                                                                  uint32_t num_tiles) {
    for (uint32_t tile = next_tile(work); tile < num_tiles; tile = next_tile(work)) {
        uint32_t i, j;
        const bool valid = tile_pixel(tile, threadIdx.x & 31, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;
        const RayState r = make_ray(mk3(cam.eye[0], cam.eye[1], cam.eye[2]), primary_dir(cam, i, j), 1e16f, -1);
        uint32_t nv = 0, nt = 0, leaf = 1;
        const Hit h = shader_trace(r, valid, tr, 1u, &nv, &nt, &leaf);
        if (valid) {
            const size_t p = (size_t)j * cam.width + i;
            store_hit(hits + p, h);
            leaves[p] = leaf;
            if (stats) {
                stats[2 * p] = nv;
                stats[2 * p + 1] = nt;
            }
        }
    }
}

__global__ void __launch_bounds__(kTraceThreads) k_shader_shade(TreeRef tr, const float* __restrict__ soup,
                                                                rt_camera cam, float lx, float ly, float lz,
                                                                const rt_hit* __restrict__ prim,
                                                                const uint32_t* __restrict__ leaves,
                                                                uint8_t* __restrict__ vis, rt_hit* __restrict__ mirror,
                                                                uint32_t* __restrict__ sstats,
                                                                uint32_t* __restrict__ mstats, uint32_t* work,
                                                                uint32_t num_tiles) {
    for (uint32_t tile = next_tile(work); tile < num_tiles; tile = next_tile(work)) {
        uint32_t i, j;
        const bool valid = tile_pixel(tile, threadIdx.x & 31, cam.width, cam.height, &i, &j);
        if (!valid) i = j = 0;
        const size_t p = (size_t)j * cam.width + i;
        int4 ph = make_int4(-1, 0, 0, 0);
        if (valid) ph = __ldg(reinterpret_cast<const int4*>(prim + p));
        const ShadeRays s = shade_rays(soup, cam, lx, ly, lz, ph, valid, i, j, mirror != nullptr);
        const uint32_t start = (valid && s.has) ? __ldg(leaves + p) : 1u;
        uint32_t snv = 0, snt = 0, mnv = 0, mnt = 0;
        if (vis) {  // uniform across the grid
            const Hit sh = shader_trace(s.shadow, valid && s.cast, tr, start, &snv, &snt, nullptr);
            if (valid) vis[p] = vis_code(s.has, s.cast, sh.id >= 0);
        }
        if (mirror) {
            Hit mh = shader_trace(s.mirror, valid && s.has, tr, start, &mnv, &mnt, nullptr);
            if (!s.has) {
                mh.id = -2; mh.u = -1.0f; mh.v = -1.0f; mh.t = 0.0f;
            }
            if (valid) store_hit(mirror + p, mh);
        }
        if (valid) {
            if (sstats) { sstats[2 * p] = snv; sstats[2 * p + 1] = snt; }
            if (mstats) { mstats[2 * p] = mnv; mstats[2 * p + 1] = mnt; }
        }
    }
}

}  // namespace

extern "C" rt_status rt_trace_frame_shader_order(rt_ctx* ctx, const rt_lbvh* l, const rt_camera* cam,
                                                 const float light[3], rt_hit* d_primary, uint8_t* d_vis,
                                                 rt_hit* d_mirror, uint32_t* d_primary_stats,
                                                 uint32_t* d_shadow_stats, uint32_t* d_mirror_stats) {
    rt_status s = check_trace_args(ctx, l, cam, "rt_trace_frame_shader_order");
    if (s != RT_OK) return s;
    if (!light || !d_primary) return rt_fail(ctx, RT_ERR_INVALID, "rt_trace_frame_shader_order: null argument");
    if ((d_vis || d_mirror) && !l->src_tris)
        return rt_fail(ctx, RT_ERR_INVALID, "rt_trace_frame_shader_order: no triangle soup bound");
    const size_t px = (size_t)cam->width * cam->height;
    // the primary leaves live in the third segment of the shading lists
    if ((s = ensure_shade_lists(ctx, const_cast<rt_lbvh*>(l), px)) != RT_OK) return s;
    uint32_t* leaves = l->s_lists + 2 * l->s_pixels;
    TreeRef tr;  // the reference's walk runs over the heap
    tr.compact = false;
    tr.tri_base = 0;
    tr.nodes = l->nodes;
    tr.num_nodes = l->num_nodes;
    tr.tris = l->sorted_tris;
    tr.n = l->n;
    tr.err = ctx->d_err;
    const uint32_t tiles = pixel_tiles(cam);
    if ((s = reset_work(ctx, kWorkPrimary)) != RT_OK) return s;
    k_shader_primary<<<persistent_blocks(ctx, k_shader_primary, kTraceThreads, tiles), kTraceThreads, 0, ctx->stream>>>(
        tr, *cam, d_primary, leaves, d_primary_stats, ctx->d_work + kWorkPrimary, tiles);
    RT_CHECK_LAUNCH(ctx, "k_shader_primary");
    if (d_vis || d_mirror) {
        if ((s = reset_work(ctx, kWorkSecondary)) != RT_OK) return s;
        k_shader_shade<<<persistent_blocks(ctx, k_shader_shade, kTraceThreads, tiles), kTraceThreads, 0,
                         ctx->stream>>>(tr, l->src_tris, *cam, light[0], light[1], light[2], d_primary, leaves, d_vis,
                                        d_mirror, d_shadow_stats, d_mirror_stats, ctx->d_work + kWorkSecondary, tiles);
        RT_CHECK_LAUNCH(ctx, "k_shader_shade");
    }
    return RT_OK;
}

// ---------------------------------------------------------------------------
// Batched trace: primary + shadow rays of every pixel of every scene of an
// rt_batch.  A work item is one 8 x 4 tile of one scene; warps take `grab`
// consecutive items per increment of one work counter, so the scenes with
// the costliest rays never hold the grid back.  The primary pass lists the
// pixels that cast a shadow ray (with the ray and its start node, the
// primary leaf) and the lane-refill kernel traces them, lanes of one warp
// walking different scenes: in the tile pass only one lane in seven had a
// shadow ray to trace.  Without a list the tile pass traces them itself.
namespace {

struct BatchTraceArgs {
    const float* soup;
    const rt_camera* cams;
    const float* lights;
    rt_hit* hits;
    uint8_t* vis;
    uint32_t S, width, height, tiles_per_scene, grab, order;
};

// The shadow-ray list of a batched trace.
struct BatchListArgs {
    uint32_t* lists;
    uint32_t cap;
    uint32_t* counts;
    float4* rays;
    uint32_t* starts;
};

// Primary rays of a batch, an 8 x 4 tile of one scene per warp at a time.  LIST:
// the shadow rays are listed; else they are traced here (a.vis set) or not
// cast (a.vis null).
constexpr int kBatchSteps = 6;  // 256 random soups: 4: 9.42 ms a frame, 6: 9.36, 8: 9.38, 12: 9.61

template <bool LIST>
__device__ __forceinline__ void batch_trace_body(const BatchTraceArgs& a, const BatchListArgs& la, const TreeRef& tr0,
                                                 const BatchTrees& bt, uint32_t* work) {
    mark_records(tr0);
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    const uint32_t total = a.S * a.tiles_per_scene;
    const uint32_t lane = threadIdx.x & 31;
    const size_t px = (size_t)a.width * a.height;
    for (;;) {
        uint32_t g0 = 0;
        if (lane == 0) g0 = atomicAdd(work, a.grab);
        g0 = __shfl_sync(0xffffffffu, g0, 0);
        if (g0 >= total) break;
        const uint32_t g1 = min(total, g0 + a.grab);
        for (uint32_t g = g0; g < g1; ++g) {
            const uint32_t s = a.order ? g % a.S : g / a.tiles_per_scene;
            const uint32_t tile = a.order ? g / a.S : g % a.tiles_per_scene;
            TreeRef tr = tr0;
            scene_tree(tr, bt, s);
            const uint32_t toff = tr.tri_base;
            const rt_camera cam = a.cams[s];
            uint32_t i, j;
            const bool valid = tile_pixel(tile, lane, a.width, a.height, &i, &j);
            if (!valid) i = j = 0;
            const RayState r = make_ray(mk3(cam.eye[0], cam.eye[1], cam.eye[2]), primary_dir(cam, i, j), 1e16f, -1);
            w.start(valid, r, tr, 1u, stack, Walk::tile_by_heap(valid, r, tr));
            while (__any_sync(0xffffffffu, w.have)) w.round<kPoolMin, false>(tr, kBatchSteps, stack);
            const Hit h = w.hit();
            const uint32_t leaf = w.b.leaf;
            const size_t p = (size_t)j * a.width + i;
            if (valid) store_hit(a.hits + s * px + p, h);
            if (LIST) {  // the shadow ray (restarting at the primary leaf) goes to the list
                const int4 ph = make_int4(h.id, __float_as_int(h.u), __float_as_int(h.v), __float_as_int(h.t));
                const ShadeLists sl{a.soup + 9 * (size_t)toff, __ldg(a.lights + 3 * s), __ldg(a.lights + 3 * s + 1),
                                    __ldg(a.lights + 3 * s + 2), a.vis, nullptr, la.lists, la.cap, la.counts,
                                    la.rays, la.starts};
                shade_setup_pixel(sl, cam, ph, valid, i, j, s * px + p, h.id >= 0 ? leaf : 1u);
            } else if (a.vis) {  // uniform across the grid; the shadow ray restarts at the primary leaf
                const int4 ph = make_int4(h.id, __float_as_int(h.u), __float_as_int(h.v), __float_as_int(h.t));
                const ShadeRays sr = shade_rays(a.soup + 9 * (size_t)toff, cam, __ldg(a.lights + 3 * s),
                                                __ldg(a.lights + 3 * s + 1), __ldg(a.lights + 3 * s + 2), ph, valid, i, j,
                                                false);
                w.start(valid && sr.cast, sr.shadow, tr, h.id >= 0 ? leaf : 1u, stack);
                while (__any_sync(0xffffffffu, w.have)) w.round<kPoolMin, false>(tr, kBatchSteps, stack, true);
                if (valid) a.vis[s * px + p] = vis_code(sr.has, sr.cast, sr.cast && w.b.id >= 0);
            }
        }
    }
}

// Blocks of 256 threads per SM (48 and 64 registers; unbounded 80): the scenes of a large
// batch do not fit the caches, and more warps hide that (256 scenes at 256 x 256
// 9.88 ms a frame unbounded, 8.59 with four, 8.38 with five, 8.34 with six; primary
// rays only, 64 scenes, 1,453, 1,178, 1,112 and 1,135 us); with few tiles a warp the spills
// cost more (16 scenes at 128 x 128 601, 602, 620 and 639 us).
bool many_tiles(const rt_ctx* ctx, uint64_t tiles) { return tiles > 8ull * 32u * (uint32_t)ctx->num_sms; }

template <int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS) k_batch_trace(BatchTraceArgs a, TreeRef tr, BatchTrees bt, uint32_t* work) {
    grid_dep_wait();
    const BatchListArgs none = {nullptr, 0u, nullptr, nullptr, nullptr};
    batch_trace_body<false>(a, none, tr, bt, work);
}

template <int BLOCKS>
__global__ void __launch_bounds__(256, BLOCKS) k_batch_list(BatchTraceArgs a, BatchListArgs la, TreeRef tr, BatchTrees bt,
                                                            uint32_t* work) {
    grid_dep_wait();
    batch_trace_body<true>(a, la, tr, bt, work);
}

}  // namespace

extern "C" rt_status rt_batch_set_views(rt_ctx* ctx, rt_batch* b, const rt_camera* h_cams, const float* h_lights) {
    if (!ctx) return RT_ERR_INVALID;
    if (!b || !h_cams || !h_lights) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_views: null argument");
    const uint32_t w = h_cams[0].width, h = h_cams[0].height;
    if (w == 0 || h == 0 || (uint64_t)w * h * b->S > (1ull << 34))
        return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_views: bad image size %ux%u", w, h);
    for (uint32_t s = 1; s < b->S; ++s)
        if (h_cams[s].width != w || h_cams[s].height != h)
            return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_views: scene %u is %ux%u, scene 0 is %ux%u", s,
                           h_cams[s].width, h_cams[s].height, w, h);
    RT_CHECK_CUDA(ctx, cudaMemcpyAsync(b->cams, h_cams, sizeof(rt_camera) * b->S, cudaMemcpyHostToDevice, ctx->stream));
    RT_CHECK_CUDA(ctx, cudaMemcpyAsync(b->lights, h_lights, sizeof(float) * 3 * b->S, cudaMemcpyHostToDevice,
                                       ctx->stream));
    // the shadow-ray list: one entry per pixel of the batch at most
    const uint64_t cap = (uint64_t)w * h * b->S;
    if (cap > b->s_cap && cap <= (1ull << 31)) {
        if (b->graph_refs > 0)
            return rt_fail(ctx, RT_ERR_CAPACITY,
                           "rt_batch_set_views: the shadow-ray list cannot grow while a captured frame uses it");
        RT_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (b->s_lists) cudaFree(b->s_lists);
        if (b->s_rays) cudaFree(b->s_rays);
        b->s_lists = nullptr;
        b->s_rays = nullptr;
        b->s_cap = 0;
        RT_CHECK_CUDA(ctx, cudaMalloc((void**)&b->s_lists, 2 * sizeof(uint32_t) * cap));
        RT_CHECK_CUDA(ctx, cudaMalloc((void**)&b->s_rays, 2 * sizeof(float4) * cap));
        b->s_cap = (uint32_t)cap;
    }
    b->width = w;
    b->height = h;
    return RT_OK;
}

extern "C" rt_status rt_batch_set_tuning(rt_ctx* ctx, rt_batch* b, const rt_batch_tuning* t) {
    if (!ctx) return RT_ERR_INVALID;
    if (!b || !t) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_tuning: null argument");
    if (t->threads != 64 && t->threads != 128 && t->threads != 256)
        return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_tuning: threads must be 64, 128 or 256");
    if (t->grab < 1 || t->grab > 16) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_tuning: grab must be in [1, 16]");
    if (t->order > 1) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_tuning: order must be 0 or 1");
    if (t->blocks_per_sm > 64) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_set_tuning: blocks_per_sm above 64");
    b->tuning = *t;
    return RT_OK;
}

extern "C" rt_status rt_batch_get_tuning(const rt_batch* b, rt_batch_tuning* t) {
    if (!b || !t) return RT_ERR_INVALID;
    *t = b->tuning;
    return RT_OK;
}

extern "C" rt_status rt_batch_trace(rt_ctx* ctx, const rt_batch* b, rt_hit* d_hits, uint8_t* d_vis) {
    if (!ctx) return RT_ERR_INVALID;
    if (!b || !d_hits) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_trace: null argument");
    if (!b->built) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_trace: the batch has not been built");
    if (b->width == 0) return rt_fail(ctx, RT_ERR_INVALID, "rt_batch_trace: no views set (rt_batch_set_views)");
    const uint64_t cap = (uint64_t)b->width * b->height * b->S;
    const bool listed = d_vis && b->s_cap >= cap && cap > 0;
    uint32_t* counts = ctx->d_work + kShadeCounts;
    uint64_t reset = word_bit(ctx, ctx->d_work + kWorkBatch);
    if (listed)
        reset |= word_bit(ctx, ctx->d_work + kWorkShade) | word_bit(ctx, counts) | word_bit(ctx, counts + 1);
    rt_status s = reset_words(ctx, reset, records_of(ctx, b));
    if (s != RT_OK) return s;
    TreeRef tr;  // the batch's arrays; heap, tnodes, tri_base and n are set per scene
    memset(&tr, 0, sizeof(tr));
    tr.tris = b->sorted_tris;
    tr.leaf_of = b->leaf_of;
    tr.num_heap = 1u << b->depth;
    tr.num_tnodes = tr.num_heap / 2;
    tr.records_valid = b->counters + 7;
    tr.err = ctx->d_err;
    const BatchTrees bt{b->nodes, b->tnodes, b->tri_off, b->depth, b->width * b->height};
    BatchTraceArgs a;
    a.soup = b->src_tris;
    a.cams = b->cams;
    a.lights = b->lights;
    a.hits = d_hits;
    a.vis = d_vis;
    a.S = b->S;
    a.width = b->width;
    a.height = b->height;
    a.tiles_per_scene = ((b->width + 7) / 8) * ((b->height + 3) / 4);
    a.grab = b->tuning.grab;
    a.order = b->tuning.order;
    const BatchListArgs la = {b->s_lists, (uint32_t)cap, counts, b->s_rays, b->s_lists + cap};
    const int threads = (int)b->tuning.threads;
    const uint64_t items = (uint64_t)a.S * a.tiles_per_scene;
    const auto list = many_tiles(ctx, items) ? k_batch_list<5> : k_batch_list<4>;
    const auto trace = many_tiles(ctx, items) ? k_batch_trace<5> : k_batch_trace<4>;
    int per_sm = 0;
    const cudaError_t oe = listed ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, list, threads, 0)
                                  : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trace, threads, 0);
    if (oe != cudaSuccess || per_sm < 1) per_sm = 1;
    if (b->tuning.blocks_per_sm) per_sm = std::min(per_sm, (int)b->tuning.blocks_per_sm);
    const uint64_t need = (items * 32 + threads - 1) / threads;
    const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)per_sm * ctx->num_sms, need));
    if (listed)
        launch_pdl(list, blocks, threads, 0, ctx->stream, a, la, tr, bt, ctx->d_work + kWorkBatch);
    else
        launch_pdl(trace, blocks, threads, 0, ctx->stream, a, tr, bt, ctx->d_work + kWorkBatch);
    RT_CHECK_LAUNCH(ctx, listed ? "k_batch_list" : "k_batch_trace");
    if (!listed) return RT_OK;
    Spill none;
    memset(&none, 0, sizeof(none));
    int shade_per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&shade_per_sm, k_walk_shade<true>, kTraceThreads, 0) != cudaSuccess ||
        shade_per_sm < 1)
        shade_per_sm = 1;
    launch_pdl(k_walk_shade<true>, (uint32_t)shade_per_sm * ctx->num_sms, kTraceThreads, 0, ctx->stream, tr, d_vis,
               (rt_hit*)nullptr, (uint32_t*)nullptr, (const uint32_t*)b->s_lists, (uint32_t)cap, (const uint32_t*)counts,
               (const float4*)b->s_rays, (const uint32_t*)(b->s_lists + cap), ctx->d_work + kWorkShade, none,
               (uint32_t*)nullptr, bt);
    RT_CHECK_LAUNCH(ctx, "k_walk_shade");
    return RT_OK;
}
