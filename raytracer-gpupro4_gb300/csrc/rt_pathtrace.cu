// rt_pathtrace.cu -- path-traced GI and its adjoint on sm_103a.
//
// Forward: the GI branch of the reference (CSPrimaryRays.hlsl:23-34,63 and
// CSComputeColorGI.hlsl:19-238 with the progressive factors of
// cbGlobalIllumination, ConstantBuffers.h:85-110), one lane per pixel with
// its path state in registers (path regeneration, below) instead of a
// 48-byte ray / 24-byte hit round trip through global memory per segment.
// Per segment: closest hit, the walk started at the previous hit's leaf
// (CSIntersections.hlsl:32); on a hit acc += (1/(n+1) * beta) * Le,
// beta *= albedo, new direction
// cosine-distributed about the facing geometric normal; on a miss
// acc += (1/(n+1) * beta) * sky.  Sampling uses one PCG32 stream per
// (pixel, sample) and Malley's method, so every operation is an IEEE
// +,-,*,/ or sqrt and the image matches the CPU rendering bit for bit.
//
// Adjoint: the same paths are replayed (nothing is stored between the
// passes); for a path with throughputs beta_s, albedos a_s and radiances E_s,
// dC/da_j = beta_j * G_j with G_j = E_{j+1} + a_{j+1} * G_{j+1}.
#include "rt_traverse.cuh"

using namespace rt;

namespace {

constexpr int kPtThreads = 128;
constexpr int kMaxSeg = 16;

struct Pcg32 {
    uint64_t state, inc;
    __device__ __forceinline__ uint32_t next() {
        const uint64_t old = state;
        state = old * 6364136223846793005ULL + inc;
        const uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u);
        const uint32_t rot = (uint32_t)(old >> 59u);
        return (xs >> rot) | (xs << ((0u - rot) & 31u));
    }
    __device__ __forceinline__ void seed(uint64_t initstate, uint64_t initseq) {
        state = 0u;
        inc = (initseq << 1u) | 1u;
        next();
        state += initstate;
        next();
    }
    __device__ __forceinline__ float uniform() { return fmul((float)(next() >> 8), 1.0f / 16777216.0f); }
};

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ void pt_seed(Pcg32& g, uint64_t seed, uint64_t pixel, uint32_t sample) {
    const uint64_t s = splitmix64(seed + 0x9E3779B97F4A7C15ULL * (pixel * 65536ULL + sample + 1ULL));
    g.seed(s, pixel);
}

// Malley's method + the orthonormal basis of Duff et al. (JCGT 2017).
__device__ __forceinline__ f3 cosine_dir(Pcg32& g, f3 n) {
    float x = 0.0f, y = 0.0f, r2 = 0.0f;
    for (int k = 0; k < 64; ++k) {
        x = fsub(fmul(2.0f, g.uniform()), 1.0f);
        y = fsub(fmul(2.0f, g.uniform()), 1.0f);
        r2 = fadd(fmul(x, x), fmul(y, y));
        if (r2 <= 1.0f) break;
        x = 0.0f; y = 0.0f; r2 = 0.0f;
    }
    const float z = fsqrt(fsub(1.0f, r2));
    const float sign = copysignf(1.0f, n.z);
    const float a = fdiv(-1.0f, fadd(sign, n.z));
    const float b = fmul(fmul(n.x, n.y), a);
    const f3 T = mk3(fadd(1.0f, fmul(fmul(fmul(sign, n.x), n.x), a)), fmul(sign, b), fmul(-sign, n.x));
    const f3 B = mk3(b, fadd(sign, fmul(fmul(n.y, n.y), a)), -n.y);
    return mk3(fadd(fadd(fmul(T.x, x), fmul(B.x, y)), fmul(n.x, z)),
               fadd(fadd(fmul(T.y, x), fmul(B.y, y)), fmul(n.y, z)),
               fadd(fadd(fmul(T.z, x), fmul(B.z, y)), fmul(n.z, z)));
}

__device__ __forceinline__ f3 facing_normal(const float* __restrict__ soup, int id, f3 d) {
    const float* tp = soup + 9 * (size_t)id;
    const f3 A = mk3(__ldg(tp), __ldg(tp + 1), __ldg(tp + 2));
    const f3 B = mk3(__ldg(tp + 3), __ldg(tp + 4), __ldg(tp + 5));
    const f3 C = mk3(__ldg(tp + 6), __ldg(tp + 7), __ldg(tp + 8));
    f3 N = normalize3(cross3(sub3(B, A), sub3(C, A)));
    if (dot3(N, d) > 0.0f) N = mk3(-N.x, -N.y, -N.z);
    return N;
}

struct PathParams {
    rt_camera cam;
    uint32_t spp, bounces;
    uint64_t seed;
    float sky[3];
    uint32_t n0;  // first sample index (samples 0 .. n0-1 are already in the image)
};

// Walk counts of the counting variant (rt_pathtrace_counted), per lane.
struct PathCounts {
    uint32_t segments = 0, boxes = 0, tris = 0, hits = 0;
};

// Path regeneration.  A warp's lanes each hold one path (a sample of a
// pixel, or a pixel whose samples follow one another, see launch_pathtrace)
// and trace it one segment at a time.  A lane whose walk has ended waits until
// kPtShadeLanes of the warp's have; those then shade, bounce or take the next
// path from the work counter, and start their next walks together while the
// other lanes keep theirs, so no lane waits for the longest walk of its warp.
// Of 2 to 16 lanes 10 was best (shading and the walk's start cost about 1,100
// instructions whatever the lanes).  Paths are handed out in 8 x 4 pixel
// tiles, lanes of one grab taking consecutive pixels.
constexpr int kPtShadeLanes = 10;
constexpr int kPtSteps = 8;  // expansions between two leaf phases (5: 26.1 ms, 7: 23.5, 8: 23.5, 10: 24.1)
// Blocks per SM: 56 registers and nine blocks where the paths fill the GPU
// (23.9 ms; eight: 24.5, seven: 26.1), 128 and four where they don't (0.70 ms a
// 256 x 256 image; eight: 0.76).
constexpr int kPtBlocks = 9, kPtSmallBlocks = 4;

struct PathLane {
    bool live = false;           // holds a path
    uint32_t i = 0, j = 0;       // the pixel
    uint32_t n = 0;              // the sample being traced
    uint32_t s = 0;              // its segment
    Pcg32 g;
    f3 o, d;
    int exclude = -1;
    uint32_t start = 1u;         // restart node of the segment's walk
    float fact = 0.0f;           // 1 / (n + 1)
    float keep = 0.0f;           // n / (n + 1)
    float beta[3];
};

// Sample n of the lane's pixel: its stream and camera ray (the GI branch of
// CSPrimaryRays.hlsl:23-34 with a sub-pixel jitter).
__device__ __forceinline__ void begin_sample(PathLane& L, const PathParams& P) {
    pt_seed(L.g, P.seed, (uint64_t)L.j * P.cam.width + L.i, L.n);
    const float inv = fdiv(1.0f, (float)P.cam.height);
    const float jx = fsub(fmul(2.0f, L.g.uniform()), 1.0f);
    const float jy = fsub(fmul(2.0f, L.g.uniform()), 1.0f);
    const float x = fmul(fadd((float)(2 * (int)L.i + 1 - (int)P.cam.width), jx), inv);
    const float y = -fmul(fadd((float)(2 * (int)L.j + 1 - (int)P.cam.height), jy), inv);
    L.d = camera_dir(P.cam, x, y);
    L.o = mk3(P.cam.eye[0], P.cam.eye[1], P.cam.eye[2]);
    L.exclude = -1;
    L.start = 1u;
    L.s = 0;
    L.beta[0] = L.beta[1] = L.beta[2] = 1.0f;
    L.keep = fdiv((float)L.n, (float)(L.n + 1));
    L.fact = fdiv(1.0f, (float)(L.n + 1));
}

// Next ray of a path that hit triangle `id` at t (not its last segment):
// origin at the hit, a cosine-distributed direction about the facing
// normal, the walk restarted at the hit's leaf.
__device__ __forceinline__ void bounce(PathLane& L, const float* __restrict__ soup, int id, float t, uint32_t leaf) {
    const f3 N = facing_normal(soup, id, L.d);
    L.o = mk3(fadd(L.o.x, fmul(t, L.d.x)), fadd(L.o.y, fmul(t, L.d.y)), fadd(L.o.z, fmul(t, L.d.z)));
    L.d = cosine_dir(L.g, N);
    L.exclude = id;
    L.start = leaf;
    ++L.s;
}

// Warp-aggregated grab of paths for the idle lanes (all lanes call): path
// p is sample first + (p / 32) % per of pixel p % 32 of tile p / (32 per).
// Returns true for a lane that took a pixel inside the image.
__device__ __forceinline__ bool grab_path(PathLane& L, const PathParams& P, uint32_t first, uint32_t per, uint32_t* work,
                                          uint32_t total, bool& drained) {
    constexpr uint32_t kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t idle = __ballot_sync(kFull, !L.live);
    if (drained || idle == 0u) return false;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(work, (uint32_t)__popc(idle));
    base = __shfl_sync(kFull, base, 0);
    if (base >= total || total - base <= (uint32_t)__popc(idle)) drained = true;
    const uint32_t k = base + __popc(idle & ((1u << lane) - 1u));
    if (!((idle >> lane) & 1u) || base >= total || k >= total) return false;
    const uint32_t tile = (k >> 5) / per;
    uint32_t i, j;
    if (!tile_pixel(tile, k & 31u, P.cam.width, P.cam.height, &i, &j)) return false;
    L.i = i;
    L.j = j;
    L.n = first + ((k >> 5) - tile * per);
    L.live = true;
    return true;
}

// Whether the lanes whose walks have ended go on now (uniform): enough of
// them, or nobody left walking.
__device__ __forceinline__ bool shade_now(bool walking, bool live, bool drained) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t w = __ballot_sync(kFull, walking);
    const uint32_t held = drained ? __ballot_sync(kFull, live) : kFull;
    return w == 0u || __popc(held & ~w) * 32 >= __popc(held) * kPtShadeLanes;
}

// The radiance terms of samples traced apart: term (sample, segment, pixel)
// = (1 / (n + 1) * beta) * Le, and how many segments each sample has.
struct PathTerms {
    float* terms;       // [spp][segments][pixels][3]
    uint8_t* segments;  // [spp][pixels]
};

// Per segment: closest hit; on a hit acc += (1/(n+1) * beta) * Le, beta *=
// albedo; on a miss acc += (1/(n+1) * beta) * sky.  TERMS: a path is one
// sample, and its terms are stored for k_fold_terms; otherwise a path is a
// pixel with all its samples.
template <bool TERMS, int BLOCKS>
__global__ void __launch_bounds__(kPtThreads, BLOCKS) k_pathtrace(
    TreeRef tr, const float* __restrict__ soup, const float* __restrict__ albedo, const float* __restrict__ emission,
    PathParams P, float4* __restrict__ image, uint32_t* work, uint32_t num_tiles, PathTerms T) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t per = TERMS ? P.spp : 1u, total = num_tiles * 32u * per;
    const size_t px = (size_t)P.cam.width * P.cam.height;
    mark_records(tr);
    PathLane L;
    L.o = mk3(0.f, 0.f, 0.f);
    L.d = mk3(0.f, 0.f, 1.f);
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    float acc[3] = {0.0f, 0.0f, 0.0f};
    bool drained = false;
    for (;;) {
        if (shade_now(w.have, L.live, drained)) {
            bool fresh = false;  // a new segment to walk
            if (L.live && !w.have) {
                bool ended = w.b.id < 0;
                float le[3] = {P.sky[0], P.sky[1], P.sky[2]};
                if (!ended)
                    for (int c = 0; c < 3; ++c) le[c] = __ldg(emission + 3 * (size_t)w.b.id + c);
                const size_t p = (size_t)L.j * P.cam.width + L.i;
                float* term = TERMS ? T.terms + 3 * (((size_t)(L.n - P.n0) * (P.bounces + 1u) + L.s) * px + p) : nullptr;
                for (int c = 0; c < 3; ++c) {
                    const float x = fmul(fmul(L.fact, L.beta[c]), le[c]);
                    if (TERMS) term[c] = x;
                    else acc[c] = fadd(acc[c], x);
                }
                if (!ended) {
                    for (int c = 0; c < 3; ++c)
                        L.beta[c] = fmul(L.beta[c], __ldg(albedo + 3 * (size_t)w.b.id + c));
                    ended = L.s == P.bounces;
                    if (!ended) bounce(L, soup, w.b.id, w.b.t, tr.compact ? 1u : w.b.leaf);
                }
                fresh = !ended;
                if (ended) {
                    if (TERMS) {
                        T.segments[(size_t)(L.n - P.n0) * px + p] = (uint8_t)(L.s + 1u);
                        L.live = false;
                    } else if (++L.n == P.n0 + P.spp) {
                        image[p] = make_float4(acc[0], acc[1], acc[2], 1.0f);
                        L.live = false;
                    } else {
                        begin_sample(L, P);
                        for (int c = 0; c < 3; ++c) acc[c] = fmul(acc[c], L.keep);
                        fresh = true;
                    }
                }
            }
            if (grab_path(L, P, P.n0, per, work, total, drained)) {
                begin_sample(L, P);
                if (!TERMS) {
                    acc[0] = acc[1] = acc[2] = 0.0f;
                    if (P.n0 > 0) {  // continue the progressive mean the image holds
                        const float4 prev = image[(size_t)L.j * P.cam.width + L.i];
                        acc[0] = prev.x;
                        acc[1] = prev.y;
                        acc[2] = prev.z;
                    }
                    for (int c = 0; c < 3; ++c) acc[c] = fmul(acc[c], L.keep);
                }
                fresh = true;
            }
            w.start(fresh, make_ray(L.o, L.d, 1e16f, L.exclude), tr, L.start, stack);
            if (!__any_sync(kFull, L.live)) {
                if (drained) break;
                continue;
            }
        }
        w.round<kPathPoolMin, false>(tr, kPtSteps, stack);
    }
}

// The progressive mean over samples n0 .. n0 + spp - 1 from their terms: the
// same sequence of fp32 operations as tracing them one after another.
__global__ void __launch_bounds__(256) k_fold_terms(PathTerms T, uint32_t px, uint32_t segs, uint32_t n0, uint32_t spp,
                                                    float4* __restrict__ image) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= px) return;
    float acc[3] = {0.0f, 0.0f, 0.0f};
    if (n0 > 0) {
        const float4 prev = image[p];
        acc[0] = prev.x;
        acc[1] = prev.y;
        acc[2] = prev.z;
    }
    for (uint32_t m = 0; m < spp; ++m) {
        const uint32_t n = n0 + m;
        const float keep = fdiv((float)n, (float)(n + 1));
        for (int c = 0; c < 3; ++c) acc[c] = fmul(acc[c], keep);
        const uint32_t ns = T.segments[(size_t)m * px + p];
        for (uint32_t s = 0; s < ns; ++s) {
            const float* term = T.terms + 3 * (((size_t)m * segs + s) * px + p);
            for (int c = 0; c < 3; ++c) acc[c] = fadd(acc[c], __ldg(term + c));
        }
    }
    image[p] = make_float4(acc[0], acc[1], acc[2], 1.0f);
}

// The counting variant: each walk in the order whose box and triangle tests
// are counted (traverse), a warp's lanes together; sums the walk counts into
// counts[4] (64-bit).
__global__ void __launch_bounds__(kPtThreads) k_pathtrace_counted(
    TreeRef tr, const float* __restrict__ soup, const float* __restrict__ albedo, const float* __restrict__ emission,
    PathParams P, float4* __restrict__ image, uint32_t* work, uint32_t num_tiles, unsigned long long* counts) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t total = num_tiles * 32u;
    PathCounts cnt;
    PathLane L;
    L.o = mk3(0.f, 0.f, 0.f);
    L.d = mk3(0.f, 0.f, 1.f);
    float acc[3] = {0.0f, 0.0f, 0.0f};
    bool drained = false;
    for (;;) {
        if (grab_path(L, P, P.n0, 1u, work, total, drained)) {
            begin_sample(L, P);
            acc[0] = acc[1] = acc[2] = 0.0f;
            if (P.n0 > 0) {
                const float4 prev = image[(size_t)L.j * P.cam.width + L.i];
                acc[0] = prev.x;
                acc[1] = prev.y;
                acc[2] = prev.z;
            }
            for (int c = 0; c < 3; ++c) acc[c] = fmul(acc[c], L.keep);
        }
        if (!__any_sync(kFull, L.live)) {
            if (drained) break;
            continue;
        }
        const RayState r = make_ray(L.o, L.d, 1e16f, L.exclude);
        uint32_t nb = 0, nt = 0, leaf = 1u;
        const Hit h = trace_ray<true>(r, L.live, tr, false, &nb, &nt, nullptr, nullptr, L.start, &leaf);
        if (!L.live) continue;
        cnt.segments += 1;
        cnt.boxes += nb;
        cnt.tris += nt;
        cnt.hits += (h.id >= 0) ? 1u : 0u;
        bool ended = h.id < 0;
        float le[3] = {P.sky[0], P.sky[1], P.sky[2]};
        if (!ended)
            for (int c = 0; c < 3; ++c) le[c] = __ldg(emission + 3 * (size_t)h.id + c);
        for (int c = 0; c < 3; ++c) acc[c] = fadd(acc[c], fmul(fmul(L.fact, L.beta[c]), le[c]));
        if (!ended) {
            for (int c = 0; c < 3; ++c) L.beta[c] = fmul(L.beta[c], __ldg(albedo + 3 * (size_t)h.id + c));
            ended = L.s == P.bounces;
            if (!ended) bounce(L, soup, h.id, h.t, leaf);
        }
        if (ended) {
            if (++L.n == P.n0 + P.spp) {
                image[(size_t)L.j * P.cam.width + L.i] = make_float4(acc[0], acc[1], acc[2], 1.0f);
                L.live = false;
            } else {
                begin_sample(L, P);
                for (int c = 0; c < 3; ++c) acc[c] = fmul(acc[c], L.keep);
            }
        }
    }
    unsigned long long v[4] = {cnt.segments, cnt.boxes, cnt.tris, cnt.hits};
    for (int q = 0; q < 4; ++q) {
        for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_xor_sync(kFull, v[q], off);
        if ((threadIdx.x & 31) == 0 && v[q]) atomicAdd(counts + q, v[q]);
    }
}

// Adjoint by path replay: the same paths as k_pathtrace (same streams, same
// hits), one sample a path; a lane records the triangles its sample hits, and
// when the sample ends runs the backward recurrence G_j = E_{j+1} + a_{j+1}
// G_{j+1} over them with the sample's weight in the final mean.
__global__ void __launch_bounds__(kPtThreads, kPtBlocks) k_pathtrace_adjoint(
    TreeRef tr, const float* __restrict__ soup,
    const float* __restrict__ albedo, const float* __restrict__ emission, PathParams P,
    const float4* __restrict__ dimage, float* __restrict__ dalbedo, double* dle_sum,
    uint32_t* work, uint32_t num_tiles, uint32_t first, uint32_t per) {
    constexpr uint32_t kFull = 0xffffffffu;
    const uint32_t total = num_tiles * 32u * per;
    PathLane L;
    L.o = mk3(0.f, 0.f, 0.f);
    L.d = mk3(0.f, 0.f, 1.f);
    float dle[3] = {0.0f, 0.0f, 0.0f};
    int seg[kMaxSeg];
    int ns = 0;
    mark_records(tr);
    Walk w;
    w.clear();
    uint2 stack[kStackSize];
    bool drained = false;
    for (;;) {
        if (shade_now(w.have, L.live, drained)) {
            bool fresh = false, ending = false;
            const bool missed = w.b.id < 0;
            if (L.live && !w.have) {
                if (!missed) seg[ns++] = w.b.id;
                if (!missed && L.s != P.bounces) {
                    bounce(L, soup, w.b.id, w.b.t, tr.compact ? 1u : w.b.leaf);
                    fresh = true;
                } else {
                    ending = true;
                }
            }
            const int rounds = __reduce_max_sync(kFull, ending ? ns : 0);
            float gw[3] = {0.0f, 0.0f, 0.0f}, beta[kMaxSeg][3], G[3] = {0.0f, 0.0f, 0.0f};
            if (ending) {
                const float4 g4 = __ldg(dimage + (size_t)L.j * P.cam.width + L.i);
                // weight of sample n in the progressive mean after the call
                float wn = 1.0f / (float)(L.n + 1);
                for (uint32_t m = L.n + 1; m < P.n0 + P.spp; ++m) wn *= (float)m / (float)(m + 1);
                gw[0] = g4.x * wn;
                gw[1] = g4.y * wn;
                gw[2] = g4.z * wn;
                beta[0][0] = beta[0][1] = beta[0][2] = 1.0f;
                for (int q = 0; q + 1 < ns; ++q)
                    for (int c = 0; c < 3; ++c) beta[q + 1][c] = beta[q][c] * __ldg(albedo + 3 * (size_t)seg[q] + c);
                if (missed)
                    for (int c = 0; c < 3; ++c) G[c] = P.sky[c];
            }
            for (int q = rounds - 1; q >= 0; --q) {
                const bool on = ending && q < ns;
                float da[3] = {0.0f, 0.0f, 0.0f};
                if (on) {
                    const float* al = albedo + 3 * (size_t)seg[q];
                    const float* le = emission + 3 * (size_t)seg[q];
                    const float l0 = __ldg(le), l1 = __ldg(le + 1), l2 = __ldg(le + 2);
                    const bool emitter = (l0 != 0.0f) || (l1 != 0.0f) || (l2 != 0.0f);
                    const float lev[3] = {l0, l1, l2};
                    for (int c = 0; c < 3; ++c) {
                        da[c] = gw[c] * beta[q][c] * G[c];
                        if (emitter) dle[c] += gw[c] * beta[q][c];
                        G[c] = lev[c] + __ldg(al + c) * G[c];
                    }
                }
                // the lanes that hit one triangle are summed first: fewer roundings than an
                // atomic each
                uint32_t peers = __match_any_sync(kFull, on ? seg[q] : -1 - (int)(threadIdx.x & 31));
                const uint32_t lane = threadIdx.x & 31;
                const bool leader = (peers & ((1u << lane) - 1u)) == 0u;
                uint32_t rank = __popc(peers & ((1u << lane) - 1u));
                peers &= 0xfffffffeu << lane;
                while (__any_sync(kFull, peers != 0u)) {
                    const int next = __ffs(peers);  // the next lane of the triangle that still holds a sum
                    for (int c = 0; c < 3; ++c) {
                        const float t = __shfl_sync(kFull, da[c], next ? next - 1 : (int)lane);
                        if (next) da[c] += t;
                    }
                    peers &= __ballot_sync(kFull, (rank & 1u) == 0u);
                    rank >>= 1;
                }
                if (on && leader)
                    for (int c = 0; c < 3; ++c)
                        if (da[c] != 0.0f) atomicAdd(dalbedo + 3 * (size_t)seg[q] + c, da[c]);
            }
            if (ending) {
                ns = 0;
                L.live = false;
            }
            if (grab_path(L, P, first, per, work, total, drained)) {
                ns = 0;
                begin_sample(L, P);
                fresh = true;
            }
            w.start(fresh, make_ray(L.o, L.d, 1e16f, L.exclude), tr, L.start, stack);
            if (!__any_sync(kFull, L.live)) {
                if (drained) break;
                continue;
            }
        }
        w.round<kPathPoolMin, false>(tr, kPtSteps, stack);
    }
    // emitter gradient: a block's sum and the sum over the blocks in FP64 (an FP32 atomic a block:
    // 4.2e-7 from the FP64 gradient at 128 x 96 and 8 samples, an atomic a warp of whole pixels
    // 2.3e-7, this 3.5e-8, in the same time)
    __shared__ double s_dle[kPtThreads / 32][3];
    for (int c = 0; c < 3; ++c) {
        double v = dle[c];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFull, v, off);
        if ((threadIdx.x & 31) == 0) s_dle[threadIdx.x >> 5][c] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int q = 0; q < kPtThreads / 32; ++q) v += s_dle[q][threadIdx.x];
        if (v != 0.0) atomicAdd(dle_sum + threadIdx.x, v);
    }
}

// The call's emitter gradient, rounded once (by the last block of the launches instead, behind a
// fence: 300 us of 20,000 at 512 x 512 and 8 samples).
__global__ void k_fold_emitter(const double* __restrict__ sum, float* __restrict__ demission) {
    const double v = sum[threadIdx.x];
    if (v != 0.0) demission[threadIdx.x] += (float)v;
}

rt_status pt_args(rt_ctx* ctx, const rt_lbvh* l, const float* a, const float* e, const rt_camera* cam,
                  const rt_pt_params* p, PathParams* out, const char* who) {
    if (!ctx) return RT_ERR_INVALID;
    if (!l || !a || !e || !cam || !p) return rt_fail(ctx, RT_ERR_INVALID, "%s: null argument", who);
    if (l->n == 0 || !l->src_tris) return rt_fail(ctx, RT_ERR_INVALID, "%s: the LBVH has not been built", who);
    if (cam->width == 0 || cam->height == 0) return rt_fail(ctx, RT_ERR_INVALID, "%s: empty image", who);
    if (p->spp == 0 || p->bounces + 1 > (uint32_t)kMaxSeg)
        return rt_fail(ctx, RT_ERR_INVALID, "%s: spp must be > 0 and bounces < %d", who, kMaxSeg);
    if ((uint64_t)p->first_sample + p->spp > 65535u)  // the per-pixel streams are seeded with pixel * 65536 + sample
        return rt_fail(ctx, RT_ERR_INVALID, "%s: first_sample + spp must stay below 65536", who);
    out->cam = *cam;
    out->spp = p->spp;
    out->bounces = p->bounces;
    out->seed = p->seed;
    out->n0 = p->first_sample;
    for (int c = 0; c < 3; ++c) out->sky[c] = p->sky[c];
    return RT_OK;
}

uint32_t px_tiles(const rt_camera* cam) {
    return (uint32_t)(((cam->width + 7) / 8) * ((cam->height + 3) / 4));
}

}  // namespace

TreeRef tree_ref(const rt_ctx* ctx, const rt_lbvh* l);

// The term buffers for as many of the call's samples as fit (0: trace each
// pixel's samples one after another).  Never in a stream capture: a graph must
// not hold a buffer that a later call may replace.
static uint32_t ensure_terms(rt_ctx* ctx, size_t px, uint32_t tiles, uint32_t segs, uint32_t spp, PathTerms* T) {
    const size_t sample = px * ((size_t)segs * 12 + 1);
    // the path counter holds 2^31 of them a launch
    const uint32_t m = (uint32_t)std::min<size_t>({spp, ctx->terms_limit / sample, ((size_t)1 << 31) / (32 * (size_t)tiles)});
    if (m < 2) return 0;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return 0;
    }
    const size_t need = m * sample;
    if (need > ctx->terms_bytes) {
        if (ctx->d_terms && cudaStreamSynchronize(ctx->stream) != cudaSuccess) return 0;
        // an allocation would break another thread's stream capture in the global mode
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (ctx->d_terms) cudaFree(ctx->d_terms);
        ctx->d_terms = nullptr;
        ctx->terms_bytes = 0;
        const bool ok = cudaMalloc((void**)&ctx->d_terms, need) == cudaSuccess;
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (!ok) {
            ctx->d_terms = nullptr;
            cudaGetLastError();
            return 0;
        }
        ctx->terms_bytes = need;
    }
    T->terms = ctx->d_terms;
    T->segments = reinterpret_cast<uint8_t*>(ctx->d_terms + 3 * (size_t)m * segs * px);
    return m;
}

static rt_status launch_pathtrace(rt_ctx* ctx, const rt_lbvh* l, const float* d_albedo, const float* d_emission,
                                  const rt_camera* cam, const rt_pt_params* p, float* d_image,
                                  unsigned long long* d_counts, const char* who) {
    PathParams P;
    rt_status s = pt_args(ctx, l, d_albedo, d_emission, cam, p, &P, who);
    if (s != RT_OK) return s;
    if (!d_image) return rt_fail(ctx, RT_ERR_INVALID, "%s: null image", who);
    const uint32_t tiles = px_tiles(cam);
    const size_t px = (size_t)cam->width * cam->height;
    float4* image = reinterpret_cast<float4*>(d_image);
    uint32_t* work = ctx->d_work + kWorkPath;
    if (d_counts) {
        if ((s = reset_work(ctx, kWorkPath)) != RT_OK) return s;
        k_pathtrace_counted<<<persistent_blocks(ctx, k_pathtrace_counted, kPtThreads, tiles), kPtThreads, 0,
                              ctx->stream>>>(tree_ref(ctx, l), l->src_tris, d_albedo, d_emission, P, image, work, tiles,
                                             d_counts);
        RT_CHECK_LAUNCH(ctx, "k_pathtrace_counted");
        return RT_OK;
    }
    // Several samples a pixel: each traced as a path of its own, their terms
    // folded in order afterwards.  With a pixel's samples on one lane the last
    // pixels of a 1024 x 1024 x 4 image kept single lanes busy for 15 % of the time,
    // and a smaller image could not fill the GPU.
    const uint32_t segs = P.bounces + 1u;
    PathTerms T = {nullptr, nullptr};
    const uint32_t chunk = P.spp > 1 ? ensure_terms(ctx, px, tiles, segs, P.spp, &T) : 0u;
    auto launch = [&](auto kernel, uint32_t per) {
        kernel<<<persistent_blocks(ctx, kernel, kPtThreads, tiles * per), kPtThreads, 0, ctx->stream>>>(
            tree_ref(ctx, l), l->src_tris, d_albedo, d_emission, P, image, work, tiles, T);
    };
    if (chunk == 0u) {
        if ((s = reset_work_and_records(ctx, kWorkPath, l)) != RT_OK) return s;
        if ((uint64_t)tiles * 32u <= (uint64_t)ctx->num_sms * kPtSmallBlocks * kPtThreads) launch(k_pathtrace<false, kPtSmallBlocks>, 1u);
        else launch(k_pathtrace<false, kPtBlocks>, 1u);
        RT_CHECK_LAUNCH(ctx, "k_pathtrace");
        return RT_OK;
    }
    for (uint32_t done = 0; done < p->spp; done += P.spp) {
        P.n0 = p->first_sample + done;
        P.spp = std::min(chunk, p->spp - done);
        if ((s = reset_work_and_records(ctx, kWorkPath, l)) != RT_OK) return s;
        if ((uint64_t)tiles * 32u * P.spp <= (uint64_t)ctx->num_sms * kPtSmallBlocks * kPtThreads)
            launch(k_pathtrace<true, kPtSmallBlocks>, P.spp);
        else
            launch(k_pathtrace<true, kPtBlocks>, P.spp);
        RT_CHECK_LAUNCH(ctx, "k_pathtrace");
        k_fold_terms<<<(uint32_t)((px + 255) / 256), 256, 0, ctx->stream>>>(T, (uint32_t)px, segs, P.n0, P.spp, image);
        RT_CHECK_LAUNCH(ctx, "k_fold_terms");
    }
    return RT_OK;
}

extern "C" rt_status rt_pathtrace(rt_ctx* ctx, const rt_lbvh* l, const float* d_albedo, const float* d_emission,
                                  const rt_camera* cam, const rt_pt_params* p, float* d_image) {
    return launch_pathtrace(ctx, l, d_albedo, d_emission, cam, p, d_image, nullptr, "rt_pathtrace");
}

extern "C" rt_status rt_pathtrace_counted(rt_ctx* ctx, const rt_lbvh* l, const float* d_albedo,
                                          const float* d_emission, const rt_camera* cam, const rt_pt_params* p,
                                          float* d_image, unsigned long long* d_counts) {
    if (!d_counts) return ctx ? rt_fail(ctx, RT_ERR_INVALID, "rt_pathtrace_counted: null counts") : RT_ERR_INVALID;
    return launch_pathtrace(ctx, l, d_albedo, d_emission, cam, p, d_image, d_counts, "rt_pathtrace_counted");
}

extern "C" rt_status rt_pathtrace_adjoint(rt_ctx* ctx, const rt_lbvh* l, const float* d_albedo,
                                          const float* d_emission, const rt_camera* cam, const rt_pt_params* p,
                                          const float* d_dimage, float* d_dalbedo, float* d_demission) {
    PathParams P;
    rt_status s = pt_args(ctx, l, d_albedo, d_emission, cam, p, &P, "rt_pathtrace_adjoint");
    if (s != RT_OK) return s;
    if (!d_dimage || !d_dalbedo || !d_demission) return rt_fail(ctx, RT_ERR_INVALID, "rt_pathtrace_adjoint: null buffer");
    const uint32_t tiles = px_tiles(cam);
    // a sample of a pixel is a path; the path counter holds 2^31 of them a launch
    const uint32_t most = std::max(1u, ctx->paths_limit / std::max(32u, tiles * 32u));
    double* sum = reinterpret_cast<double*>(ctx->d_words + kEmitterSum);
    for (uint32_t done = 0; done < P.spp; done += most) {
        const uint32_t per = std::min(most, P.spp - done);
        if ((s = reset_work_and_records(ctx, kWorkAdjoint, l, done == 0u ? 0x3full << kEmitterSum : 0ull)) != RT_OK) return s;
        k_pathtrace_adjoint<<<persistent_blocks(ctx, k_pathtrace_adjoint, kPtThreads, tiles * per), kPtThreads, 0,
                              ctx->stream>>>(tree_ref(ctx, l), l->src_tris, d_albedo, d_emission, P,
                                             reinterpret_cast<const float4*>(d_dimage), d_dalbedo, sum,
                                             ctx->d_work + kWorkAdjoint, tiles, P.n0 + done, per);
        RT_CHECK_LAUNCH(ctx, "k_pathtrace_adjoint");
    }
    k_fold_emitter<<<1, 3, 0, ctx->stream>>>(sum, d_demission);
    RT_CHECK_LAUNCH(ctx, "k_fold_emitter");
    return RT_OK;
}
