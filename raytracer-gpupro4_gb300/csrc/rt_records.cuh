// rt_records.cuh -- the trace records (TraceNode in rt_internal.cuh).
//
// Walk (rt_traverse.cuh) reads the tree through them.  A build leaves them
// invalid (counters[7] = 0) and a trace call makes them before its first
// pass, in the kernel that zeroes the call's counters: callers that only build
// do not pay for them (10 us of 312 at 2.1 M triangles, wherever in the build
// they were written).  The trace kernel that follows on the stream marks them
// valid, so a mark always means complete records; two streams that trace a
// fresh tree at once both write the same values.
#pragma once
#include "rt_internal.cuh"

namespace rt {

// The grid of a tree with bounds [mn, mx]: G, E.  Bounds that are NaN make E NaN, and
// every ray reads the heap.
__device__ __forceinline__ float4 trace_grid(const float mn[3], const float mx[3]) {
    const float d[3] = {fsub(mx[0], mn[0]), fsub(mx[1], mn[1]), fsub(mx[2], mn[2])};
    const float E = isnan(d[0]) || isnan(d[1]) || isnan(d[2]) ? NAN : fmaxf(d[0], fmaxf(d[1], d[2]));
    return make_float4(fsub(mn[0], E), fsub(mn[1], E), fsub(mn[2], E), E);
}
__device__ __forceinline__ void store_trace_grid(TraceNode* tnodes, float4 g, bool by_slot) {
    *reinterpret_cast<float4*>(tnodes) = make_float4(g.x, g.y, g.z, by_slot ? -fabsf(g.w) : fabsf(g.w));
}

// One axis of a child's box; rE = 1 / E.  The lowest bit of the grid step is
// `bit` when bit >= 0.  box_enter ignores an axis whose bounds are both NaN (a soup with
// NaN vertices), so such an axis gets the whole line; and it takes the bounds in
// either order (an imported tree may hold them so).
__device__ __forceinline__ uint32_t trace_box_word(float mn, float mx, float G, float E, float rE, int bit) {
    if (!isfinite(mn) || !isfinite(mx)) return 0x7e808000u | (uint32_t)max(bit, 0);  // half-extent 2^126
    const float q = fminf(fmaxf(rintf((0.5f * mn + 0.5f * mx - (G + E)) * rE * 32768.0f), 0.0f), 32767.0f);
    uint32_t step = (uint32_t)q;
    if (bit >= 0) step = (step & ~1u) | (uint32_t)bit;
    const float X = fmaf(E, 1.0f + (float)step * (1.0f / 32768.0f), G);  // the centre, within 2^-24 |X|
    float e = fmaxf(fmaxf(__fsub_ru(mx, X), __fsub_ru(X, mn)), fmaxf(__fsub_ru(X, mx), __fsub_ru(mn, X)));
    e = __fadd_ru(e, __fmaf_ru(fabsf(X), 1.0f / 4194304.0f, E * (1.0f / 65536.0f)));  // 256 u E, and X's own error
    e = __fmul_ru(__fmul_ru(e, rE), 1.0f + 1.0f / 1048576.0f);                        // rE and k are rounded
    const uint32_t bits = __float_as_uint(fmaxf(e, 0.0f));
    uint32_t w = (bits & 0xffff0000u) | 0x8000u | step;
    if (w < bits) w += 0x10000u;
    return w;
}

// Record of internal node h split on `axis` (0 x, 1 y, 2 z) with children of
// boxes [llo, lhi], [rlo, rhi] and words lw, rw.
__device__ __forceinline__ void store_trace_node(TraceNode* tnodes, uint32_t h, const float* llo, const float* lhi,
                                                 const float* rlo, const float* rhi, uint32_t lw, uint32_t rw, int axis,
                                                 float4 g) {
    const float rE = fdiv(1.0f, g.w);
    uint4* p = reinterpret_cast<uint4*>(tnodes + h);
    p[0] = make_uint4(trace_box_word(llo[0], lhi[0], g.x, g.w, rE, axis & 1),
                      trace_box_word(llo[1], lhi[1], g.y, g.w, rE, axis >> 1),
                      trace_box_word(llo[2], lhi[2], g.z, g.w, rE, -1), trace_box_word(rlo[0], rhi[0], g.x, g.w, rE, -1));
    p[1] = make_uint4(trace_box_word(rlo[1], rhi[1], g.y, g.w, rE, -1), trace_box_word(rlo[2], rhi[2], g.z, g.w, rE, -1),
                      lw, rw);
}

// Trace record of internal node h from its children's heap records.
__device__ __forceinline__ void trace_node_of(uint32_t h, const rt_node* nodes, uint32_t num_nodes, TraceNode* tnodes,
                                              float4 g) {
    const float4* p = reinterpret_cast<const float4*>(nodes + 2u * h);
    const float4 l0 = __ldg(p), l1 = __ldg(p + 1), r0 = __ldg(p + 2), r1 = __ldg(p + 3);
    const int lpc = __float_as_int(l1.z), rpc = __float_as_int(r1.z), field = __ldg(&nodes[h].prim_count) & 3;
    const float llo[3] = {l0.x, l0.y, l0.z}, lhi[3] = {l0.w, l1.x, l1.y}, rlo[3] = {r0.x, r0.y, r0.z},
                rhi[3] = {r0.w, r1.x, r1.y};
    store_trace_node(tnodes, h, llo, lhi, rlo, rhi,
                     (lpc & 4) ? leaf_word(2u * h, (uint32_t)__float_as_int(l1.w), (uint32_t)(lpc >> 3)) : 0u,
                     (rpc & 4) ? leaf_word(2u * h + 1u, (uint32_t)__float_as_int(r1.w), (uint32_t)(rpc >> 3)) : 0u,
                     field == 0 ? 2 : field - 1, g);  // the field is one past the split axis
}

// What make_records needs of a tree (tiles = 0: no records).
struct Records {
    const uint32_t* valid;
    const uint2* units;      // the emission's leaves, kTreeTile slots per tile
    const uint32_t* counts;  // leaves of each tile
    uint32_t tiles;          // tiles that have blocks of their own
    const uint32_t* built;   // tiles of the tree when the kernel runs (nullptr: `tiles`): a captured call may be
                             // replayed over a later build
    const rt_node* nodes;
    uint32_t num_nodes;
    TraceNode* tnodes;
    uint32_t slices;         // blocks that share a tile
    uint32_t scene_depth;    // a batch's heap depth (a leaf is named by scene << 23 | heap slot); 0: one tree
};

// Few tiles are shared by two blocks each, about two blocks per SM.
inline uint32_t record_slices(uint32_t tiles, int num_sms) {
    return std::max(1u, std::min(2u, 2u * (uint32_t)num_sms / std::max(1u, tiles)));
}
inline Records records_of(const rt_ctx* ctx, const rt_lbvh* l) {
    const uint32_t tiles = std::max(1u, l->rec_tiles);
    return Records{l->counters + 7, reinterpret_cast<const uint2*>(l->keys_alt),
                   l->item_counts + 6 * (size_t)l->emit_tiles_cap, l->tnodes ? tiles : 0u, l->counters + 8, l->nodes,
                   l->num_nodes, l->tnodes, l->rec_tiles ? record_slices(tiles, ctx->num_sms) : 1u, 0u};
}
inline Records records_of(const rt_ctx* ctx, const rt_batch* b) {
    const uint32_t tiles = (b->total + kTreeTile - 1) / kTreeTile;
    return Records{b->counters + 7, reinterpret_cast<const uint2*>(b->keys), b->item_counts + 6 * (size_t)tiles,
                   b->tnodes ? tiles : 0u, nullptr, b->nodes, 1u << b->depth, b->tnodes,
                   record_slices(tiles, ctx->num_sms), b->depth};
}

// The records of a slice of a tile's leaves (block q of tiles * slices).  There is
// one internal node per two neighbouring leaves of a tree, their lowest common
// ancestor: a thread takes a leaf and the one before it.
__device__ __forceinline__ void make_records(const Records& R, uint32_t block) {
    if (*R.valid) return;  // uniform
    const bool batch = R.scene_depth != 0u;
    const uint32_t tiles = R.built ? *R.built : R.tiles;
    for (uint32_t tile = block / R.slices; tile < tiles; tile += R.tiles) {
        const uint32_t cnt = min(__ldg(R.counts + tile), (uint32_t)kTreeTile);
        uint32_t prev = 0u;  // thread 0 of slice 0: the last leaf of the tiles before, by its warp (a leaf may span many)
        if (cnt && block % R.slices == 0u && threadIdx.x < 32u) {
            for (uint32_t top = tile; top > 0u; top -= min(top, 32u)) {
                const uint32_t c = threadIdx.x < top ? min(__ldg(R.counts + (top - 1u - threadIdx.x)), (uint32_t)kTreeTile) : 0u;
                const uint32_t m = __ballot_sync(0xffffffffu, c != 0u);
                if (!m) continue;
                const int w = __ffs(m) - 1;
                prev = __ldg(&R.units[(size_t)(top - 1u - w) * kTreeTile + __shfl_sync(0xffffffffu, c, w) - 1u].x);
                break;
            }
        }
        for (uint32_t i = (block % R.slices) * blockDim.x + threadIdx.x; i < cnt; i += R.slices * blockDim.x) {
            uint32_t b = __ldg(&R.units[(size_t)tile * kTreeTile + i].x);
            uint32_t a = i ? __ldg(&R.units[(size_t)tile * kTreeTile + i - 1].x) : prev;
            const rt_node* nodes = R.nodes;
            TraceNode* tnodes = R.tnodes;
            if (batch) {
                const uint32_t sc = b >> 23;
                nodes += (size_t)sc << R.scene_depth;
                tnodes += (size_t)sc << (R.scene_depth - 1u);
                a = (a >> 23) == sc ? a & 0x7fffffu : 0u;
                b &= 0x7fffffu;
            }
            const float4* p = reinterpret_cast<const float4*>(nodes + 1);
            const float4 r0 = __ldg(p), r1 = __ldg(p + 1);
            const float mn[3] = {r0.x, r0.y, r0.z}, mx[3] = {r0.w, r1.x, r1.y};
            const float4 g = trace_grid(mn, mx);
            if (a == 0u) {  // the tree's first leaf
                store_trace_grid(tnodes, g, false);
                continue;
            }
            const int da = 31 - __clz(a), db = 31 - __clz(b), dm = min(da, db);
            const uint32_t x = (a >> (da - dm)) ^ (b >> (db - dm));
            if (b == 0u || x == 0u) continue;  // only after a failed sort
            const uint32_t h = (a >> (da - dm)) >> (32 - __clz(x));
            if (h != 0u && 2u * h + 1u < R.num_nodes) trace_node_of(h, nodes, R.num_nodes, tnodes, g);
        }
    }
}

}  // namespace rt
