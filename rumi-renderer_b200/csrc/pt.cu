// Wavefront path tracer with next-event estimation.
//
// The reference's PathTracer::Trace(w, h, ...) (src/Integrator/pathtracer.cpp:117-354)
// walks forward recording a vertex chain, then accumulates backwards
//     L_k = A_k * (direct_k + vol_k * fr_k * L_{k+1} * cos_k / Average(pdf_wi_k * pdf_path_k))
// (A_k: medium factor of the arriving segment).  Expanding the recursion gives the
// forward estimator used here: L = sum_k beta_k * direct_k with
//     beta_{k+1} = beta_k * vol_k * fr_k * cos_k / Average(pdf_wi_k * pdf_path_k),
// which lets every bounce run as independent kernels over queues of rays:
//
//   generate  camera rays (Pinhole::CastViewRay, the reference's pixel sampler)
//   extend    closest hit of every queued ray            (persistent, work-fetching)
//   shade     medium free flight, emission, BSDF sample, NEE; compacts the next
//             bounce's rays and this bounce's shadow rays with block-aggregated atomics
//   sort      large waves: an order of the next rays by origin and direction
//   shadow    any-hit test of the shadow rays; adds their contribution
//   resolve   per-pixel sum of the samples in sample order (NaN samples dropped and
//             counted, src/Scene/scene.cpp:229-241)
//
// Random numbers: Philox4x32-10 keyed by the seed, counter (path, bounce, group); a
// path's stream does not depend on the wave size or launch order.
#include "renderer.h"
#include "traverse.cuh"
#include "shading.cuh"
#include "camera.cuh"
#include "optional_block.h"
#include <map>
#include <mutex>
#include <utility>
#include <vector>
#include <type_traits>

namespace rumi {

static constexpr int TRACE_THREADS = 128;
// Minimum resident traversal blocks per SM: 8 caps the extend / shadow kernels at 64
// registers (32 warps per SM instead of 28 at their natural 72); measured 5% faster per
// frame on the 1M-triangle workload.  10 and 12 spill and are slower.  The any-hit kernel
// alone (55 registers at 8) measured 83.2 / 84.9 / 122.0 ms per frame at 9 / 10 / 12
// blocks against 83.6 at 8.
#ifndef RUMI_TRACE_MIN_BLOCKS
#define RUMI_TRACE_MIN_BLOCKS 8
#endif
#ifndef RUMI_EXTEND_MIN_BLOCKS
#define RUMI_EXTEND_MIN_BLOCKS RUMI_TRACE_MIN_BLOCKS
#endif
#ifndef RUMI_SHADOW_MIN_BLOCKS
#define RUMI_SHADOW_MIN_BLOCKS RUMI_TRACE_MIN_BLOCKS
#endif
// The default walk (SCHEME_WIDE, the speculative while-while walk over the four-wide tree) at 9
// blocks: 56 registers (a 42-byte spill in closest-hit, none in any-hit); per 1024x1024x64 frame
// 65.7 / 35.2 ms of closest-hit / any-hit against 66.7 / 36.4 at 8 and 69.9 / 35.2 at 10 (before the
// rays were ordered).
#ifndef RUMI_WW_MIN_BLOCKS
#define RUMI_WW_MIN_BLOCKS 9
#endif
// Testing a small scene's records in step (SCHEME_FEW): 64 registers without spills; 6 and 10 blocks
// are 4% slower and equal on the Cornell frame.
#ifndef RUMI_FEW_MIN_BLOCKS
#define RUMI_FEW_MIN_BLOCKS 8
#endif
static constexpr int trace_min_blocks(int mode, bool extend) {
    return mode == SCHEME_FEW    ? RUMI_FEW_MIN_BLOCKS
           : mode == SCHEME_WIDE ? RUMI_WW_MIN_BLOCKS
                                 : (extend ? RUMI_EXTEND_MIN_BLOCKS : RUMI_SHADOW_MIN_BLOCKS);
}
// 1: each bounce's any-hit launch runs on an auxiliary stream beside the next bounce's
// closest-hit launch (pt_render_in); 0: one stream, launches in order.
#ifndef RUMI_PT_OVERLAP
#define RUMI_PT_OVERLAP 1
#endif
static constexpr int STACK_SMEM = 32;
// Leaf records (the empty one included) up to which a single-node scene's rays are traced in step
// (scene_scheme; eleven would still gain).
#ifndef RUMI_FEW_RECORDS
#define RUMI_FEW_RECORDS 10
#endif
// Paths of a wave and nodes of the four-wide tree from which a wave's rays are ordered (sort_wave).
#ifndef RUMI_SORT_PATHS
#define RUMI_SORT_PATHS (1 << 22)
#endif
#ifndef RUMI_SORT_NODES
#define RUMI_SORT_NODES 64
#endif
// Rays of one bounce from which they are taken in order (in_order).
#ifndef RUMI_SORT_RAYS
#define RUMI_SORT_RAYS (1 << 21)
#endif
static constexpr int WALK_SMEM = 16;  // of the default walk (stack_entries)
static_assert(TRACE_THREADS == WW_THREADS, "the walk's shared-memory columns are one per thread");
static constexpr int DEFAULT_WALK_MODE = RUMI_WALK8 ? SCHEME_EIGHT : SCHEME_WIDE;
// Threads per block of the shading kernels; a block groups its next rays by direction, so
// the block size is also the grouping's width (128: shading 0.5 ms faster per frame,
// closest-hit 0.5 ms slower).
#ifndef RUMI_SHADE_THREADS
#define RUMI_SHADE_THREADS 256
#endif
static constexpr int SHADE_THREADS = RUMI_SHADE_THREADS;

enum { PFL_LE = 1, PFL_IN = 2 };
// A queued ray's o.w holds its path slot (bits 0-29) and its flags: bit 31 = in_object
// (read by the traversal), bit 30 = le.  Its throughput travels in the queue too
// (beta_q, same position), so shading reads and writes path state in queue order.
RUMI_D float pack_slot(int slot, unsigned fl) {
    return __int_as_float(slot | ((fl & PFL_IN) ? (int)0x80000000 : 0) | ((fl & PFL_LE) ? 0x40000000 : 0));
}
RUMI_D int slot_of(float w) { return __float_as_int(w) & 0x3fffffff; }
RUMI_D unsigned flags_of(float w) {
    const unsigned b = __float_as_uint(w);
    return ((b >> 31) ? PFL_IN : 0u) | (((b >> 30) & 1u) ? PFL_LE : 0u);
}
// counters.  The shadow queue has two sets of them (PtLaunch::sh_set, by the bounce's parity), so
// that the kernels can clear each other's without a launch for it (PtLaunch::chained).
enum { C_RAY0 = 0, C_RAY1 = 1, C_SHADOW = 2, C_FETCH_EXT = 3, C_FETCH_SH = 4, C_SHADOW1 = 5, C_FETCH_SH1 = 6, C_SORT = 7, C_NUM = 8 };
// 64-bit device statistics
enum { S_RAYS_EXT = 0, S_RAYS_SH = 1, S_NAN = 2, S_NODES = 3, S_PRIMS = 4, S_NUM = 8 };

struct PtLaunch {
    DevScene s;
    int spp, max_depth;
    uint32_t k0, k1;
    int grid_d, square;
    long long path0;
    int n_paths, pix0, n_pix;
    float4 *ray[2], *hit;  // ray: two per ray (load_ray)
    float4 *sh_ray, *sh_c;
    float4 *beta_q[2], *L;  // beta_q: throughput (+ one word) in queue order, per ray buffer
    int *cnt;
    unsigned long long *stats;
    float *film;
    int refill_min;
    // chained: the bounce's kernels keep the counters and statistics themselves.  Closest hit of
    // bounce b clears the queue count and the shadow set that shading of b fills (their last
    // readers, shading of b - 1 and the any-hit launch of b - 2, are done), shading clears the
    // closest-hit work counter and counts its rays, any hit counts its own.  0: pt_reset and
    // pt_finish do all that.
    int chained, sh_set;
    // ordered frames (GROUP_FRAME): sort_perm lists the bounce's rays in traversal order where
    // `sorted` (the camera's rays are in order as they are) and they are many (in_order)
    int sorted;
    int *sort_bins, *sort_base, *sort_perm;
    int2 *sort_key;
    // multi-scene batches (scenes == nullptr: the single scene s)
    const DevScene *scenes;
    const long long *scene_path0;  // n_scenes + 1 prefix: first global path of each scene
    const long long *scene_pix0;   // n_scenes + 1 prefix: first global pixel of each scene
    const uint32_t *scene_key;     // Philox key per scene (2 words)
    const int *scene_spp;
    int n_scenes;
    int *slot_scene;               // scene of each wave slot
    // path-replay adjoint (dls == nullptr: plain rendering)
    const float4 *Lt;              // per slot: the path's radiance from the first pass
    float4 *dls;                   // per slot: dLoss / d(path radiance), RGB (0 for NaN paths)
    const float *dfilm;            // dLoss / dfilm, H*W*3 in B,G,R order
    float2 *sh_s;                  // per shadow ray: (d log / d sigma coefficient, d log / d g)
    float *g_albedo;               // n_tris * 3 RGB, or nullptr
    float *g_medium;               // 7: sigma_s rgb, sigma_a rgb, g
};

// Parameter order of the medium gradient.
enum { GM_SIGMA_S = 0, GM_SIGMA_A = 3, GM_G = 6, GM_NUM = 7 };

// d/dg log p_HG(cos; g): the score of a direction drawn from (or weighted by) the
// Henyey-Greenstein phase function.
RUMI_D float hg_dlog_dg(float c, float g) {
    const float denom = 1.0f + g * g - 2.0f * g * c;
    return -2.0f * g / (1.0f - g * g) - 3.0f * (g - c) / denom;
}

// Sums `v` over the lanes of the warp that share `key` (>= 0) and adds the sums to
// base[3 * key + 0..2] with one atomic per group.  Called by all 32 lanes.
RUMI_D void warp_add3_by_key(float *base, int key, float3 v) {
    const unsigned act = __ballot_sync(0xffffffffu, key >= 0);
    if (key < 0) return;
    const unsigned grp = __match_any_sync(act, key);
    float3 acc = mk3(0.0f, 0.0f, 0.0f);
    unsigned m = grp;
    while (m) {
        const int src = __ffs(m) - 1;
        m &= m - 1;
        acc.x += __shfl_sync(grp, v.x, src);
        acc.y += __shfl_sync(grp, v.y, src);
        acc.z += __shfl_sync(grp, v.z, src);
    }
    if ((int)(threadIdx.x & 31) == __ffs(grp) - 1) {
        atomicAdd(base + 3 * key + 0, acc.x);
        atomicAdd(base + 3 * key + 1, acc.y);
        atomicAdd(base + 3 * key + 2, acc.z);
    }
}

RUMI_D float warp_sum(float x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Largest k with prefix[k] <= g (prefix has n + 1 ascending entries).
RUMI_D int find_scene(const long long *prefix, int n, long long g) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (prefix[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// A queued ray, origin and direction together: one 32-byte access, so that a queue position written
// or read by itself is one whole sector and not the halves of two.  Against two arrays, shading of
// a 1024x1024, 64 spp, depth-10 frame of a million triangles takes 20.0 ms, not 21.4, and closest
// hit and any hit 64.1 and 34.0, not 64.3 and 34.1.
RUMI_D void load_ray(const float4 *q, int i, float4 &o, float4 &d) {
    const float4 *p = q + 2 * (size_t)i;
#ifdef RUMI_HOST_BUILD
    o = p[0];
    d = p[1];
#else
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(o.x), "=f"(o.y), "=f"(o.z), "=f"(o.w), "=f"(d.x), "=f"(d.y), "=f"(d.z), "=f"(d.w)
                 : "l"(p));
#endif
}
RUMI_D void store_ray(float4 *q, int i, float4 o, float4 d) {
    float4 *p = q + 2 * (size_t)i;
#ifdef RUMI_HOST_BUILD
    p[0] = o;
    p[1] = d;
#else
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(o.x), "f"(o.y), "f"(o.z),
                 "f"(o.w), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w)
                 : "memory");
#endif
}

// warp_push to two queues by every thread of a block, with one addition to each counter per block:
// additions to one address are done one after another, about one a nanosecond, so a warp's own
// additions hold a large bounce up (shading of a 1024x1024, 64 spp, depth-10 frame of a million
// triangles 22.3 ms with an addition per warp to the shadow queue, 21.4 with one per block; a
// 333x251, 25 spp frame of a medium 1.36 and 1.32 ms with both queues).
RUMI_D void block_push2(int *count_a, bool want_a, int &a, int *count_b, bool want_b, int &b) {
#ifdef RUMI_HOST_BUILD
    a = warp_push(count_a, want_a);
    b = warp_push(count_b, want_b);
#else
    __shared__ int s_n[2], s_base[2];
    if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
    __syncthreads();
    a = warp_push(&s_n[0], want_a);
    b = warp_push(&s_n[1], want_b);
    __syncthreads();
    if (threadIdx.x < 2) {
        const int n = s_n[threadIdx.x];
        s_base[threadIdx.x] = n > 0 ? atomicAdd(threadIdx.x ? count_b : count_a, n) : 0;
    }
    __syncthreads();
    a += s_base[0];
    b += s_base[1];
#endif
}

// How shading leaves a block's next rays in the queue: as they come, grouped by direction within the
// block, or as they come with a bin and a rank in it for ordering the whole wave (pt_sort_order).
enum Group { GROUP_NONE, GROUP_BLOCK, GROUP_FRAME };

// The order of a large wave's rays: bins of origin cell (16^3 over the scene's bounds) times
// direction cell (8^3 over [-1, 1]^3), both along a Morton curve.  Rays of one bin walk the same
// nodes, so a warp's lanes diverge less and its loads fall into fewer lines.  Measured on the bounces
// of a 1024x1024, 64 spp frame of a million triangles (33, 24, 20 and 17 million rays), the queue's
// own order against these bins: closest hit 5.31, 4.57, 3.82, 3.29 and 4.68, 3.60, 2.94, 2.51 ms; and
// as shading follows the same order, any hit of the bounces 2.84, 3.38, 2.84, 2.54 and 2.84, 3.00,
// 2.29, 2.02 ms.  8^3 origin cells: 0.8 ms more per frame; 16^3 direction cells with 8^3 origins:
// 0.2 ms more.
// The low four bits of the origin cell come last, after the direction: with the whole cell first,
// rays that start in one cell (a view of a small part of the scene, a scene inside a far larger
// sphere) have 512 counters in 16 lines, and their additions wait for each other.  A 2048x2048, 4 spp,
// depth-10 frame of 1034 triangles inside a sphere of 40 times their size takes 34.1 / 25.7 / 24.9 /
// 24.2 ms with 0 / 3 / 4 / 5 such bits and 22.4 ms without the order; the frame above 104.7 / 104.5 /
// 104.9 / 105.2 ms.
#ifndef RUMI_SORT_O
#define RUMI_SORT_O 4
#endif
#ifndef RUMI_SORT_D
#define RUMI_SORT_D 3
#endif
#ifndef RUMI_SORT_LOW
#define RUMI_SORT_LOW 4
#endif
static constexpr int SORT_BINS = 1 << (3 * (RUMI_SORT_O + RUMI_SORT_D));
// Bits 0-3 of the cell of x in [0, 1] at every third bit; outside it the nearest cell, NaN the first.
RUMI_D int sort_cell(float x, int bits) {
    const int c = (int)fminf(fmaxf(x * (float)(1 << bits), 0.0f), (float)((1 << bits) - 1));
    return (c & 1) | ((c & 2) << 2) | ((c & 4) << 4) | ((c & 8) << 6);
}
RUMI_D int sort_bin(const DevScene &S, float3 o, float3 d) {
    const float4 *root = reinterpret_cast<const float4 *>(S.nodes);
    const float4 a = __ldg(root), b = __ldg(root + 1);  // lo.xyz, hi.x; hi.yz
    const int co = sort_cell((o.x - a.x) / (a.w - a.x), RUMI_SORT_O) |
                   (sort_cell((o.y - a.y) / (b.x - a.y), RUMI_SORT_O) << 1) |
                   (sort_cell((o.z - a.z) / (b.y - a.z), RUMI_SORT_O) << 2);
    const int cd = sort_cell(0.5f * d.x + 0.5f, RUMI_SORT_D) | (sort_cell(0.5f * d.y + 0.5f, RUMI_SORT_D) << 1) |
                   (sort_cell(0.5f * d.z + 0.5f, RUMI_SORT_D) << 2);
    return ((co >> RUMI_SORT_LOW) << (3 * RUMI_SORT_D + RUMI_SORT_LOW)) | (cd << RUMI_SORT_LOW) |
           (co & ((1 << RUMI_SORT_LOW) - 1));
}
// Whether the n rays of a bounce are taken in that order: in a frame of which most paths leave the
// scene the later bounces have too few for it, and the pass over all bins would cost more than their
// walk (a 2048x2048, 4 spp, depth-10 frame of 1024 triangles in the open: 3.00 ms, 3.37 when every
// bounce is ordered, 3.02 when none is).
RUMI_D bool in_order(const PtLaunch &P, int n) { return P.sorted && n >= RUMI_SORT_RAYS; }

// The chained kernels' bookkeeping, by one thread of the grid.
RUMI_D bool first_thread() { return blockIdx.x == 0 && threadIdx.x == 0; }
RUMI_D int *shadow_count(const PtLaunch &P) { return P.cnt + (P.sh_set ? C_SHADOW1 : C_SHADOW); }
RUMI_D int *shadow_fetch(const PtLaunch &P) { return P.cnt + (P.sh_set ? C_FETCH_SH1 : C_FETCH_SH); }
RUMI_D void chain_extend(const PtLaunch &P, int bounce) {
    if (P.chained && first_thread()) {
        P.cnt[(bounce & 1) ^ 1] = 0;
        *shadow_count(P) = 0;
        *shadow_fetch(P) = 0;
    }
}
RUMI_D void chain_shade(const PtLaunch &P, int bounce) {
    if (P.chained && first_thread()) {
        P.stats[S_RAYS_EXT] += (unsigned long long)P.cnt[bounce & 1];
        P.cnt[C_FETCH_EXT] = 0;
    }
}
RUMI_D void chain_shadow(const PtLaunch &P) {
    if (P.chained && first_thread()) P.stats[S_RAYS_SH] += (unsigned long long)*shadow_count(P);
}

RUMI_D int isqrt_floor(int n) {
    int d = 0;
    while ((d + 1) * (d + 1) <= n) ++d;
    return d;
}

__global__ void pt_generate(PtLaunch P) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j == 0) P.cnt[C_RAY0] = P.n_paths;
    if (j >= P.n_paths) return;
    // one call site of the sampler and camera for both forms, so a batched scene's rays
    // are bit-identical to the single-scene ones
    const DevScene *S = &P.s;
    long long pixel, path = P.path0 + j;
    int s, spp = P.spp, gd = P.grid_d;
    bool square = P.square != 0;
    uint32_t k0 = P.k0, k1 = P.k1;
    if (P.scenes) {
        const long long g = P.path0 + j;
        const int k = find_scene(P.scene_path0, P.n_scenes, g);
        S = &P.scenes[k];
        spp = P.scene_spp[k];
        const long long local = g - P.scene_path0[k];
        path = local;
        pixel = local / spp;
        s = (int)(local % spp);
        gd = isqrt_floor(spp);
        square = gd * gd == spp;
        k0 = P.scene_key[2 * k];
        k1 = P.scene_key[2 * k + 1];
        P.slot_scene[j] = k;
    } else {
        pixel = (long long)P.pix0 + j / P.spp;
        s = j % P.spp;
    }
    const int W = S->width;
    const int w = (int)(pixel % W), h = (int)(pixel / W);
    const float2 smp = pixel_sample(s, spp, gd, square, pixel, k0, k1);
    float3 o, d;
    const float2 lu = S->camera.focal_distance > 0.0f ? lens_uniforms((uint64_t)path, k0, k1) : make_float2(0.f, 0.f);
    camera_ray(S->camera, W, S->height, w, h, smp.x, smp.y, lu.x, lu.y, o, d);
    store_ray(P.ray[0], j, make_float4(o.x, o.y, o.z, pack_slot(j, PFL_LE)), make_float4(d.x, d.y, d.z, FLT_MAX));
    P.beta_q[0][j] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    P.L[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (P.dls) {
        // the film drops NaN samples (pt_resolve), so they receive no gradient
        const long long px = (long long)P.pix0 + j / P.spp;
        const float4 lt = P.Lt[j];
        const bool nan = lt.x != lt.x || lt.y != lt.y || lt.z != lt.z;
        P.dls[j] = nan ? make_float4(0.0f, 0.0f, 0.0f, 0.0f)
                       : make_float4(P.dfilm[3 * px + 2], P.dfilm[3 * px + 1], P.dfilm[3 * px + 0], 0.0f);
    }
}

__global__ void pt_reset(PtLaunch P, int bounce) {
    const int cur = bounce & 1, nxt = cur ^ 1;
    P.stats[S_RAYS_EXT] += (unsigned long long)P.cnt[cur];
    if (bounce > 0) P.stats[S_RAYS_SH] += (unsigned long long)P.cnt[C_SHADOW];
    P.cnt[nxt] = 0;
    P.cnt[C_SHADOW] = 0;
    P.cnt[C_FETCH_EXT] = 0;
    P.cnt[C_FETCH_SH] = 0;
}

__global__ void pt_finish(PtLaunch P) { P.stats[S_RAYS_SH] += (unsigned long long)P.cnt[C_SHADOW]; }

// Persistent traversal kernels: every block takes rays from the bounce's queue until it
// is empty (traverse_queue in traverse.cuh; MODE selects the scheme, see there).
// SMEM: traversal stack entries per thread kept in shared memory (deeper entries spill to
// local memory); a smaller stack leaves more of the SM's unified L1/shared storage to L1.
template <int MODE, bool STATS, int SMEM = STACK_SMEM>
__global__ void __launch_bounds__(TRACE_THREADS, trace_min_blocks(MODE, true)) pt_extend(PtLaunch P, int bounce) {
    __shared__ int stack[SMEM * TRACE_THREADS];
    const int cur = bounce & 1;
    chain_extend(P, bounce);
    const bool ordered = in_order(P, P.cnt[cur]);
    TraceStats st{0, 0};
    auto fetch = [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
        float4 o4, d4;
        load_ray(P.ray[cur], ordered ? P.sort_perm[i] : i, o4, d4);
        o = f4xyz(o4);
        d = f4xyz(d4);
        tmax = d4.w;
        in_obj = (__float_as_uint(o4.w) >> 31) != 0;
    };
    auto finish = [&](int i, const HitRec &h) {
        const int code = h.t > 0.0f ? (h.id | (h.back ? (int)0x80000000 : 0)) : -1;
        P.hit[i] = make_float4(h.t, __int_as_float(code), h.u, h.v);
    };
    traverse_queue<MODE, false, SMEM, STATS>(P.s, P.cnt[cur], &P.cnt[C_FETCH_EXT], P.refill_min, stack, fetch, finish,
                                             st);
    if (STATS) {
        atomicAdd(&P.stats[S_NODES], (unsigned long long)st.nodes);
        atomicAdd(&P.stats[S_PRIMS], (unsigned long long)st.prims);
    }
}

template <int MODE, bool ADJ = false, int SMEM = STACK_SMEM>
__global__ void __launch_bounds__(TRACE_THREADS, trace_min_blocks(MODE, false)) pt_shadow(PtLaunch P) {
    __shared__ int stack[SMEM * TRACE_THREADS];
    chain_shadow(P);
    TraceStats st{0, 0};
    float acc_sigma = 0.0f, acc_g = 0.0f;  // adjoint: score-weighted contributions
    auto fetch = [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
        float4 o4, d4;
        load_ray(P.sh_ray, i, o4, d4);
        o = f4xyz(o4);
        d = f4xyz(d4);
        tmax = d4.w;
        in_obj = false;
    };
    auto finish = [&](int i, const HitRec &h) {
        if (h.t == 0.0f) {
            const int slot = __float_as_int(P.sh_ray[2 * (size_t)i].w);
            const float4 c = P.sh_c[i];
            float4 l = P.L[slot];
            l.x += c.x; l.y += c.y; l.z += c.z;
            P.L[slot] = l;
            if (ADJ) {
                // this NEE term alone carries the shadow ray's transmittance decision
                // and (in a medium) the phase function's value at the light direction
                const float4 dl = P.dls[slot];
                const float dterm = dl.x * c.x + dl.y * c.y + dl.z * c.z;
                const float2 sc = P.sh_s[i];
                acc_sigma += sc.x * dterm;
                acc_g += sc.y * dterm;
            }
        }
    };
    traverse_queue<MODE, true, SMEM, false>(P.s, *shadow_count(P), shadow_fetch(P), P.refill_min,
                                            stack, fetch, finish, st);
    if (ADJ) {
        __syncwarp();
        acc_sigma = warp_sum(acc_sigma);
        acc_g = warp_sum(acc_g);
        if ((threadIdx.x & 31) == 0 && (acc_sigma != 0.0f || acc_g != 0.0f)) {
            for (int k = 0; k < 6; ++k) atomicAdd(&P.g_medium[k], acc_sigma);
            atomicAdd(&P.g_medium[GM_G], acc_g);
        }
    }
}

// Multi-scene batches: the default traversal scheme (speculative while-while, the walk
// rumi_render uses) with each ray's own scene, so a batched scene resolves exact-distance
// ties exactly as its single-scene render does.
template <bool ANYHIT>
__global__ void __launch_bounds__(TRACE_THREADS, trace_min_blocks(DEFAULT_WALK_MODE, !ANYHIT))
    pt_trace_multi(PtLaunch P, int bounce) {
    __shared__ int stack[WALK_SMEM * TRACE_THREADS];
    const int cur = bounce & 1;
    const int n = ANYHIT ? *shadow_count(P) : P.cnt[cur];
    int *counter = ANYHIT ? shadow_fetch(P) : &P.cnt[C_FETCH_EXT];
    if (ANYHIT)
        chain_shadow(P);
    else
        chain_extend(P, bounce);
    TraceStats st{0, 0};
    auto scene_of = [&](int i) -> const DevScene * {
        if (i < 0) return &P.scenes[0];
        const float4 o4 = (ANYHIT ? P.sh_ray : P.ray[cur])[2 * (size_t)i];
        return &P.scenes[P.slot_scene[ANYHIT ? __float_as_int(o4.w) : slot_of(o4.w)]];
    };
    auto fetch = [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
        float4 o4, d4;
        load_ray(ANYHIT ? P.sh_ray : P.ray[cur], i, o4, d4);
        o = f4xyz(o4);
        d = f4xyz(d4);
        tmax = d4.w;
        in_obj = !ANYHIT && (__float_as_uint(o4.w) >> 31) != 0;
    };
    auto finish = [&](int i, const HitRec &h) {
        if (ANYHIT) {
            if (h.t == 0.0f) {
                const int slot = __float_as_int(P.sh_ray[2 * (size_t)i].w);
                const float4 c = P.sh_c[i];
                float4 l = P.L[slot];
                l.x += c.x; l.y += c.y; l.z += c.z;
                P.L[slot] = l;
            }
        } else {
            const int code = h.t > 0.0f ? (h.id | (h.back ? (int)0x80000000 : 0)) : -1;
            P.hit[i] = make_float4(h.t, __int_as_float(code), h.u, h.v);
        }
    };
    traverse_queue_walk<ANYHIT, WALK_SMEM, false>(scene_of, n, counter, P.refill_min, stack, fetch, finish, st);
}

// Next-event estimation toward one light sample from p.  Returns false when the light
// faces away or lies outside a spot cone (Scene::VisibilityTest's facing test,
// src/Scene/scene.cpp:99-123).  wi / dist: the shadow ray; G: AreaLight::G.
RUMI_D bool nee_setup(const LightSample &ls, float3 p, float3 &wi, float &dist, float &G) {
    if (ls.is_ibl) {  // ImageBasedLight: Wi is the sampled direction, G = 1
        wi = ls.wi;
        const float3 dv = rn_sub(ls.P, p);
        dist = __fsqrt_rn(rn_dot(dv, dv));
        G = 1.0f;
        return rn_dot(wi, ls.nL) < 0.0f;
    }
    const float3 dv = ls.P - p;
    wi = normalize_ref(dv);
    dist = sqrtf(dot3(p - ls.P, p - ls.P));
    if (ls.is_delta) {
        if (dot3(-wi, ls.spot_dir) < ls.cos_cone) return false;
        G = 1.0f / (dist * dist);
        return true;
    }
    if (dot3(wi, ls.nL) >= 0.0f) return false;
    G = fmaxf(-dot3(wi, ls.nL), 0.0f) / (dist * dist);
    return true;
}

// ADJ: the replay pass of the path-replay adjoint (pt_backward).  Every path is traced a
// second time on the same random numbers; at each of its events the part of the path's
// radiance that the event influences -- Lt (the first pass's total) minus the terms
// already accumulated -- is weighted with dLoss/dradiance and with the event's score:
//   triangle albedo at a Lambertian vertex: d log / d rho = 1 / rho (per channel)
//   medium segment passed through:         log P = -avg(sigma_t) * s_max
//   medium scatter at distance s:          log p = log avg(sigma_t) - avg(sigma_t) s
//                                                  + log(1 - avg(sigma_a / sigma_t)),
//                                          weight sigma_s / sigma_t (per channel)
//   phase direction (applied at the next vertex) and NEE phase value: d log HG / d g
//   binary shadow transmittance (applied by the shadow kernel to that NEE term alone).
// Forward shading is bound by the latency of its scattered per-path loads and by instruction
// fetch, so more warps pay even for spills: a 333x251, 25 spp, depth-9 frame of a medium around a
// glass sphere shades in 1.56 / 1.43 / 1.37 ms at two / three / four blocks of 256 threads per SM
// (118, 80 and 64 registers), 1.40 ms in blocks of 128 at the same 64 registers, 1.49 ms at 48.
// The adjoint replay keeps its registers (two to four blocks: no difference).
#ifndef RUMI_SHADE_MIN_BLOCKS
#define RUMI_SHADE_MIN_BLOCKS 4
#endif
// The Whitted kernel at four blocks (64 registers): 0.29 ms of a 640x480, 9 spp, depth-10 frame's
// shading against 0.39 ms without a limit (73 registers).
#ifndef RUMI_SHADE_WHITTED_MIN_BLOCKS
#define RUMI_SHADE_WHITTED_MIN_BLOCKS 4
#endif
// LEAN: the instantiation for scenes without a medium, textures, image-based lights or
// subsurface materials (the host picks it only for those): the same code with the branches
// those features take compiled out, so the kernel holds fewer registers and instructions.
// Everything it executes is what the general instantiation executes for such a scene.
// The lean instantiation fits four blocks (64 registers, a 52-byte spill): 21.8 ms of
// shading per frame against 25.6 ms at three blocks (72 registers, no spill) and 27.9 ms for
// the general instantiation.
#ifndef RUMI_SHADE_LEAN_MIN_BLOCKS
#define RUMI_SHADE_LEAN_MIN_BLOCKS 4
#endif
template <bool ADJ, bool LEAN = false, Group GROUP = GROUP_BLOCK>
__global__ void __launch_bounds__(SHADE_THREADS, ADJ ? 1 : (LEAN ? RUMI_SHADE_LEAN_MIN_BLOCKS : RUMI_SHADE_MIN_BLOCKS))
    pt_shade(PtLaunch P, int bounce) {
    const int cur = bounce & 1, nxt = cur ^ 1;
    chain_shade(P, bounce);
    const int n = P.cnt[cur];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < n;

    bool want_next = false, want_sh = false;
    float3 nx_o = mk3(0, 0, 0), nx_d = mk3(0, 0, 0);
    unsigned nx_flags = 0;
    float3 sh_o = mk3(0, 0, 0), sh_d = mk3(0, 0, 0), sh_c = mk3(0, 0, 0);
    float sh_tmax = 0.0f;
    int slot = 0;
    float3 beta = mk3(0, 0, 0);
    float pend_g = 0.0f;                     // adjoint: score of the phase direction sampled here
    float2 sh_score = make_float2(0.0f, 0.0f);
    float gm[GM_NUM];
    int alb_key = -1;
    float3 alb_grad = mk3(0.0f, 0.0f, 0.0f);
    if (ADJ) {
#pragma unroll
        for (int k = 0; k < GM_NUM; ++k) gm[k] = 0.0f;
    }

    if (active) {
        float4 o4, d4;
        const int q = GROUP == GROUP_FRAME && in_order(P, n) ? P.sort_perm[i] : i;  // hits are in the order
        load_ray(P.ray[cur], q, o4, d4);
        const float4 hv = P.hit[i];
        slot = slot_of(o4.w);
        const DevScene *Sp = &P.s;
        uint32_t k0 = P.k0, k1 = P.k1;
        uint64_t path = (uint64_t)(P.path0 + slot);
        if (P.scenes) {
            const int sk = P.slot_scene[slot];
            Sp = &P.scenes[sk];
            k0 = P.scene_key[2 * sk];
            k1 = P.scene_key[2 * sk + 1];
            path = (uint64_t)(P.path0 + slot - P.scene_path0[sk]);
        }
        const DevScene &S = *Sp;
        const float3 o = f4xyz(o4), d = f4xyz(d4);
        const float t = hv.x;
        const bool hit = t > 0.0f;
        const int code = __float_as_int(hv.y);
        const unsigned fl = flags_of(o4.w);
        const bool le = (fl & PFL_LE) != 0, inobj = (fl & PFL_IN) != 0;
        const float4 beta4 = P.beta_q[cur][q];
        beta = f4xyz(beta4);
        // adjoint: radiance of the terms from this vertex on, and its loss weights
        float3 Lo = mk3(0.0f, 0.0f, 0.0f), dl = mk3(0.0f, 0.0f, 0.0f);
        float D = 0.0f;
        if (ADJ) {
            const float4 lt = P.Lt[slot], la = P.L[slot], d4 = P.dls[slot];
            Lo = mk3(lt.x - la.x, lt.y - la.y, lt.z - la.z);
            dl = f4xyz(d4);
            D = dot3(dl, Lo);
            gm[GM_G] += beta4.w * D;  // the direction sampled at the previous (medium) vertex
        }
        const Uniform4 U0 = path_uniforms(path, bounce, 0, k0, k1);
        const Uniform4 U1 = path_uniforms(path, bounce, 1, k0, k1);
        const bool last = bounce + 1 >= P.max_depth;
        float3 addL = mk3(0, 0, 0);
        bool done = false;

        // ---------------------------------------------- homogeneous medium
        const DevVolume &V = S.volume;
        if (!LEAN && V.present && !inobj) {
            float tn, tf;
            const float thit = hit ? t : 0.0f;
            if (volume_intersect(V, o, d, thit, tn, tf)) {
                const float smax = volume_max_distance(thit, tn, tf);
                const DistSample ds = distance_sample(V.sigma_t, V.avg_sigma_t, V.absorb, smax, U1.u[2], U1.u[3]);
                if (ADJ) {
                    const float third = 0.33333333333f;
                    if (ds.outcome == 0) {
                        const float c = -smax * third * D;
#pragma unroll
                        for (int k = 0; k < 6; ++k) gm[k] += c;
                    } else if (ds.outcome == 1) {
                        const float base = (third / V.avg_sigma_t - ds.s * third) * D;
                        const float inv1a = 1.0f / (1.0f - V.absorb);
                        const float ss[3] = {V.sigma_s.x, V.sigma_s.y, V.sigma_s.z};
                        const float sa[3] = {V.sigma_a.x, V.sigma_a.y, V.sigma_a.z};
                        const float st[3] = {V.sigma_t.x, V.sigma_t.y, V.sigma_t.z};
                        const float q[3] = {dl.x * Lo.x, dl.y * Lo.y, dl.z * Lo.z};
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float t2 = 3.0f * st[c] * st[c];
                            const float ws = ss[c] > 0.0f ? 1.0f / ss[c] - 1.0f / st[c] : 0.0f;
                            gm[GM_SIGMA_S + c] += base + sa[c] / t2 * inv1a * D + ws * q[c];
                            gm[GM_SIGMA_A + c] += base - ss[c] / t2 * inv1a * D - q[c] / st[c];
                        }
                    }
                }
                if (ds.outcome == 2) {
                    done = true;  // absorbed (pathtracer.cpp:164-167)
                } else if (ds.outcome == 1) {
                    const float3 p = o + d * (tn < 0.0f ? ds.s : tn + ds.s);
                    const float3 vol = ds.tau / ds.pdf;
                    // HomogeneousVolume::DirectLighting (homogeneousvolume.cpp:231-250)
                    if (S.n_lights > 0) {
                        // the vertex keeps the normal of the surface hit beyond the scatter
                        // point (pathtracer.cpp:154-170 moves only _p); an image-based light
                        // samples about it
                        float3 nb = mk3(0.0f, 1.0f, 0.0f);
                        if (hit && S.lights[pick_light(S, U0.u[3])].type == LIGHT_IBL) {
                            const int hid = code & 0x7fffffff;
                            nb = surface_normal(S, hid, code < 0, hv.z, hv.w, o, rn_madd(o, d, t),
                                                S.materials[prim_material(S, hid)]);
                        }
                        const LightSample ls = sample_light(S, U0.u[3], U1.u[0], U1.u[1], p, nb);
                        float3 wi;
                        float dist, G;
                        if (nee_setup(ls, p, wi, dist, G)) {
                            const Uniform4 U2 = path_uniforms(path, bounce, 2, k0, k1);
                            float smax_sh = 0.0f;
                            const float tr = volume_shadow_tr(V, p, wi, dist, U2.u[2], &smax_sh);
                            if (tr > 0.0f) {
                                if (ADJ) sh_score = make_float2(-smax_sh * 0.33333333333f, hg_dlog_dg(dot3(d, wi), V.g));
                                const float fp = V.g == 0.0f ? 1.0f / (4.0f * RUMI_PI_F) : hg_eval(dot3(d, wi), V.g);
                                const float3 direct = ls.Li * tr * V.sigma_s * fp * G * (1.0f / ls.pdf);
                                want_sh = true;
                                sh_o = p;
                                sh_d = wi;
                                sh_tmax = dist;
                                sh_c = beta * vol * direct;
                            }
                        }
                    }
                    // phase sampling; Fp / pdf = sigma_s (isotropic: the reference's
                    // Fp = sigma_s / 4 pi over Average(pdf_wi) = 1 / 4 pi)
                    float pdf_phase;
                    const float3 w = V.g == 0.0f ? isotropic_dir(d, U0.u[1], U0.u[2])
                                                 : hg_sample(d, V.g, U0.u[1], U0.u[2], pdf_phase);
                    float3 fp_over_pdf;
                    if (V.g == 0.0f) {
                        const float fp = 1.0f / (4.0f * RUMI_PI_F);
                        const float pdf = avg3(mk3(fp, fp, fp));
                        fp_over_pdf = V.sigma_s * fp * (1.0f / pdf);
                    } else {
                        fp_over_pdf = V.sigma_s;
                    }
                    beta = beta * vol * fp_over_pdf;
                    if (ADJ) pend_g = hg_dlog_dg(dot3(d, w), V.g);
                    nx_o = p;
                    nx_d = w;
                    nx_flags = 0;  // le = false, in_object = false
                    want_next = !last;
                    done = true;
                }
            }
        }

        // ---------------------------------------------------- surface
        if (!done && hit) {
            const int id = code & 0x7fffffff;
            const bool back = code < 0;
            const int mi = prim_material(S, id);
            const DevMaterial m = S.materials[mi];
            float3 p = rn_madd(o, d, t);
            float3 nrm;
            float3 albedo = m.rgb;
            if (id < S.n_tris) {
                const float4 n0 = __ldg(&S.tri_shade[3 * id]), n1 = __ldg(&S.tri_shade[3 * id + 1]),
                             n2 = __ldg(&S.tri_shade[3 * id + 2]);
                const float u = hv.z, v = hv.w;
                nrm = bary_ref(f4xyz(n0), f4xyz(n1), f4xyz(n2), u, v);  // triangle.cpp:111 (Q3)
                if (back && material_opaque(m)) nrm = -nrm;
                if (S.tri_albedo) albedo = f4xyz(__ldg(&S.tri_albedo[id]));
                if (ADJ && P.g_albedo && S.tri_albedo && m.type == MAT_MATTE) {
                    // every term from this vertex on carries the factor albedo (per channel)
                    alb_key = id;
                    alb_grad = mk3(albedo.x > 0.0f ? dl.x * Lo.x / albedo.x : 0.0f,
                                   albedo.y > 0.0f ? dl.y * Lo.y / albedo.y : 0.0f,
                                   albedo.z > 0.0f ? dl.z * Lo.z / albedo.z : 0.0f);
                }
            } else if (id < S.n_tris + S.n_rects) {
                const int r = id - S.n_tris;
                nrm = normalize_ref(cross3(f4xyz(S.rects[3 * r + 1]), f4xyz(S.rects[3 * r + 2])));
            } else {
                const float4 c = S.spheres[id - S.n_tris - S.n_rects];
                const float3 cc = f4xyz(c);
                if (m.type == MAT_EMISSIVE) {
                    const float3 oc = o - cc;
                    nrm = sqrtf(dot3(oc, oc)) > c.w ? normalize_ref(p - cc) : normalize_ref(cc - p);
                } else {
                    nrm = normalize_ref(p - cc);
                }
            }
            if (m.type == MAT_EMISSIVE) {
                // Emissive::DirectLighting (emissive.cpp:61-74) times the texture
                // (pathtracer.cpp:343-344); the path ends here.
                if (le && !inobj && -dot3(d, nrm) > 0.0f) addL = LEAN ? beta * m.le : beta * m.le * tex_pattern(S, id, p);
            } else {
                const float3 wo = -d;
                BsdfSample b;
                float3 vol_ratio = mk3(1, 1, 1), volw = mk3(1, 1, 1);
                bool walk_scatter = false, absorbed = false;
                if (!LEAN && m.type == MAT_SUBSURFACE && inobj) {
                    // Subsurface::PhaseSampling (subsurface.cpp:121-142): random walk step
                    const Uniform4 U2 = path_uniforms(path, bounce, 2, k0, k1);
                    const DistSample ws = distance_sample(m.sigma_t, m.avg_sigma_t, m.absorb, t, U2.u[0], U2.u[1]);
                    if (ws.outcome == 1) {
                        walk_scatter = true;
                        p = o + d * ws.s;
                        b.w = isotropic_dir(-wo, U0.u[1], U0.u[2]);
                        b.le = true;
                        b.go_in = true;
                        b.xi = 1.0f;
                        b.pdf_path = 1.0f;
                        b.cost = 1.0f;
                        b.pdfw = 1.0f / (4.0f * RUMI_PI_F);
                        volw = ws.tau / ws.pdf * (m.rgb * (1.0f / (4.0f * RUMI_PI_F)));
                    } else if (ws.outcome == 2) {
                        absorbed = true;
                    } else {
                        vol_ratio = ws.tau / ws.pdf;
                        b = material_sample(m, wo, nrm, U0.u[0], U0.u[1], U0.u[2]);
                    }
                } else {
                    b = material_sample(m, wo, nrm, U0.u[0], U0.u[1], U0.u[2]);
                }
                // Texture::Pattern scales everything this vertex returns, its light
                // sample and what comes after it (pathtracer.cpp:343-344)
                if (!LEAN && S.prim_tex) beta = beta * tex_pattern(S, id, p);
                if (!absorbed) {
                    // NEE: Matte::DirectLighting (matte.cpp:54-82); Glossy only on its
                    // diffuse lobe, divided by kd_pdf (glossy.cpp:92-102)
                    const bool nee = S.n_lights > 0 && !walk_scatter &&
                                     (m.type == MAT_MATTE ||
                                      (m.type == MAT_GLOSSY && m.kd != 0.0f && b.xi <= m.kd_pdf));
                    if (nee) {
                        const LightSample ls = sample_light<!LEAN>(S, U0.u[3], U1.u[0], U1.u[1], p, nrm);
                        float3 wi;
                        float dist, G;
                        if (nee_setup(ls, p, wi, dist, G)) {
                            const float3 f = albedo * RUMI_INV_PI_F * m.kd;
                            const float cost = fmaxf(dot3(wi, nrm), 0.0f);
                            float3 direct = f * ls.Li * cost * G / ls.pdf;
                            if (m.type == MAT_GLOSSY) direct = direct * (1.0f / m.kd_pdf);
                            float tr = 1.0f;
                            if (!LEAN && V.present) {
                                const Uniform4 U2 = path_uniforms(path, bounce, 2, k0, k1);
                                float smax_sh = 0.0f;
                                tr = volume_shadow_tr(V, p, wi, dist, U2.u[2], &smax_sh);
                                if (ADJ) sh_score = make_float2(-smax_sh * 0.33333333333f, 0.0f);
                            }
                            // a shadow ray whose contribution is exactly zero (the light
                            // below the surface's horizon: cos = 0) cannot change the film
                            // and is not traced; NaN and inf contributions are
                            const float3 c = beta * direct;
                            if (tr > 0.0f && (c.x != 0.0f || c.y != 0.0f || c.z != 0.0f)) {
                                want_sh = true;
                                sh_o = p;
                                sh_d = wi;
                                sh_tmax = dist;
                                sh_c = c;
                            }
                        }
                    }
                    const float3 fr = walk_scatter ? mk3(1, 1, 1)
                                                   : material_fr(m, albedo, nrm, b.w, wo, inobj, b.xi, b.pdf_path,
                                                                 t, vol_ratio);
                    const float pdf = avg3(mk3(b.pdfw * b.pdf_path, b.pdfw * b.pdf_path, b.pdfw * b.pdf_path));
                    beta = beta * volw * fr * b.cost * (1.0f / pdf);
                    nx_o = p;
                    nx_d = b.w;
                    nx_flags = (b.le ? PFL_LE : 0) | (b.go_in ? PFL_IN : 0);
                    want_next = !last;
                }
            }
        }
        if (addL.x != 0.0f || addL.y != 0.0f || addL.z != 0.0f) {
            float4 l = P.L[slot];
            l.x += addL.x; l.y += addL.y; l.z += addL.z;
            P.L[slot] = l;
        }
    }
    // GROUP_BLOCK: the next rays of this block go to the queue grouped by direction (octant x dominant
    // axis: 24 bins), in one contiguous range per block.  The traversal kernels take rays
    // in queue order, so a warp then holds rays from a few neighbouring pixels' hit points
    // that head the same way (closest-hit 2% faster per frame on the 1M-triangle
    // workload).  A path's result does not depend on its queue position.
    int kn = -1, ks = -1;
#ifdef RUMI_HOST_BUILD
    // host build (one emulated thread per block): the block's group is its one ray
    kn = want_next ? atomicAdd(&P.cnt[nxt], 1) : -1;
    ks = want_sh ? atomicAdd(shadow_count(P), 1) : -1;
#else
    if (GROUP == GROUP_BLOCK) {
        __shared__ int s_bins[32], s_shadow[2];
        if (threadIdx.x < 32) s_bins[threadIdx.x] = 0;
        if (threadIdx.x == 32) s_shadow[0] = 0;
        __syncthreads();
        int dkey = 0, drank = 0;
        if (want_next) {
            const float ax = fabsf(nx_d.x), ay = fabsf(nx_d.y), az = fabsf(nx_d.z);
            const int dom = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
            const int oct = (nx_d.x < 0.0f ? 1 : 0) | (nx_d.y < 0.0f ? 2 : 0) | (nx_d.z < 0.0f ? 4 : 0);
            dkey = oct * 3 + dom;
            drank = atomicAdd(&s_bins[dkey], 1);
        }
        ks = warp_push(&s_shadow[0], want_sh);
        __syncthreads();
        if (threadIdx.x < 32) {  // exclusive scan of the bins, then the block's range of the queue
            const int v = s_bins[threadIdx.x];
            int incl = v;
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o) incl += u;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            int base = 0;
            if (threadIdx.x == 0 && total > 0) base = atomicAdd(&P.cnt[nxt], total);
            base = __shfl_sync(0xffffffffu, base, 0);
            s_bins[threadIdx.x] = base + incl - v;
        } else if (threadIdx.x == 32) {  // and of the shadow queue
            s_shadow[1] = s_shadow[0] > 0 ? atomicAdd(shadow_count(P), s_shadow[0]) : 0;
        }
        __syncthreads();
        if (want_next) kn = s_bins[dkey] + drank;
        ks += s_shadow[1];
    } else {
        int2 key = make_int2(0, 0);
        if (GROUP == GROUP_FRAME && want_next) {
            key.x = sort_bin(P.s, nx_o, nx_d);
            key.y = atomicAdd(&P.sort_bins[key.x], 1);
        }
        block_push2(&P.cnt[nxt], want_next, kn, shadow_count(P), want_sh, ks);
        if (GROUP == GROUP_FRAME && want_next) P.sort_key[kn] = key;
    }
#endif
    if (want_next) {
        store_ray(P.ray[nxt], kn, make_float4(nx_o.x, nx_o.y, nx_o.z, pack_slot(slot, nx_flags)),
                  make_float4(nx_d.x, nx_d.y, nx_d.z, FLT_MAX));
        P.beta_q[nxt][kn] = make_float4(beta.x, beta.y, beta.z, pend_g);
    }
    if (want_sh) {
        store_ray(P.sh_ray, ks, make_float4(sh_o.x, sh_o.y, sh_o.z, __int_as_float(slot)),
                  make_float4(sh_d.x, sh_d.y, sh_d.z, sh_tmax));
        P.sh_c[ks] = make_float4(sh_c.x, sh_c.y, sh_c.z, 0.0f);
        if (ADJ) P.sh_s[ks] = sh_score;
    }
    if (ADJ) {
        warp_add3_by_key(P.g_albedo, alb_key, alb_grad);
        // medium: warp sums, then one atomic per parameter per block
        __shared__ float red[SHADE_THREADS / 32][GM_NUM];
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
        for (int k = 0; k < GM_NUM; ++k) {
            const float v = warp_sum(gm[k]);
            if (lane == 0) red[warp][k] = v;
        }
        __syncthreads();
        if (threadIdx.x < GM_NUM) {
            float v = 0.0f;
            for (int w = 0; w < SHADE_THREADS / 32; ++w) v += red[w][threadIdx.x];
            if (v != 0.0f) atomicAdd(&P.g_medium[threadIdx.x], v);
        }
    }
}

#ifndef RUMI_HOST_BUILD
// Ordering a wave's next rays, after shading has counted them by bin and given each its rank there:
// the queue range of every bin (bins in order within a block's 4096, blocks as they come), counters
// back to zero; then each ray's queue position into its place of sort_perm.  Where the rays are too
// few for the order, their bins' counters are cleared and nothing else is done.  The rays themselves stay:
// moving their 48 bytes takes 16 ms of the frame above, against 2 here and 2 in the gathers of
// closest hit and shading.
static constexpr int SORT_THREADS = 1024;
static_assert(SORT_BINS % (4 * SORT_THREADS) == 0, "one int4 of bins per thread");
__global__ void __launch_bounds__(SORT_THREADS) pt_sort_bases(PtLaunch P, int queue) {
    if (!in_order(P, P.cnt[queue])) return;
    __shared__ int s_sum[32], s_base;
    const int i = blockIdx.x * SORT_THREADS + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 v = reinterpret_cast<int4 *>(P.sort_bins)[i];
    reinterpret_cast<int4 *>(P.sort_bins)[i] = make_int4(0, 0, 0, 0);
    const int n = v.x + v.y + v.z + v.w;
    int incl = n;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int w = s_sum[lane];
        int wi = w;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += u;
        }
        s_sum[lane] = wi - w;
        if (lane == 31) s_base = wi > 0 ? atomicAdd(&P.cnt[C_SORT], wi) : 0;
    }
    __syncthreads();
    const int base = s_base + s_sum[warp] + incl - n;
    reinterpret_cast<int4 *>(P.sort_base)[i] = make_int4(base, base + v.x, base + v.x + v.y, base + v.x + v.y + v.z);
}

__global__ void pt_sort_order(PtLaunch P, int queue) {
    const int n = P.cnt[queue], first = blockIdx.x * blockDim.x + threadIdx.x;
    const bool ordered = in_order(P, n);
    if (first == 0) P.cnt[C_SORT] = 0;
    for (int i = first; i < n; i += gridDim.x * blockDim.x) {
        const int2 key = P.sort_key[i];
        if (ordered)
            P.sort_perm[P.sort_base[key.x] + key.y] = i;
        else
            P.sort_bins[key.x] = 0;
    }
}
#endif

// RayTracer::Trace (src/Integrator/raytracer.cpp:37-72), the Whitted integrator, on the
// same queues as the path tracer.  A vertex at trace depth `bounce` (the camera ray is
// depth 0; depths up to max_depth are shaded, so the host runs max_depth + 1 bounces):
//   Specular   -> Specular::GlobalIllumination: mirror ray, weight kr * colour
//                 (specular.cpp:60-75);
//   Dielectric -> Dielectric::GlobalIllumination: reflection with probability kr, else
//                 refraction with weight 1 / eta^2, eta = in_object ? eta_in / eta_out
//                 : eta_out / eta_in; a ray that goes into the object is attenuated by
//                 Beer-Lambert over the length it travels, with the absorption of the
//                 material it entered (dielectric.cpp:105-159);
//   otherwise  -> the material's DirectLighting and the walk ends: Matte next-event
//                 estimation (matte.cpp:54-82), Glossy only when its Intersection::_rand
//                 (1.0 here, nothing samples a lobe) falls on the diffuse lobe
//                 (glossy.cpp:92-102), Emissive emission when le, outside objects and
//                 front-facing (emissive.cpp:61-74), Subsurface nothing.
// No medium event: the RayTracer sends rays through a volume unattenuated; only the
// shadow ray of next-event estimation sees it (HomogeneousVolume::ShadowRayTr).  beta.w
// carries the index of the material a refracted ray entered.
__global__ void __launch_bounds__(SHADE_THREADS, RUMI_SHADE_WHITTED_MIN_BLOCKS) pt_shade_whitted(PtLaunch P, int bounce) {
    const int cur = bounce & 1, nxt = cur ^ 1;
    chain_shade(P, bounce);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = P.cnt[cur];
    const bool active = i < n;
    bool want_next = false, want_sh = false;
    float3 nx_o = mk3(0, 0, 0), nx_d = mk3(0, 0, 0);
    unsigned nx_flags = 0;
    float3 sh_o = mk3(0, 0, 0), sh_d = mk3(0, 0, 0), sh_c = mk3(0, 0, 0);
    float sh_tmax = 0.0f;
    int slot = 0, enter_mat = 0;
    float3 beta = mk3(0, 0, 0);
    if (active) {
        float4 o4, d4;
        load_ray(P.ray[cur], i, o4, d4);
        const float4 hv = P.hit[i];
        slot = slot_of(o4.w);
        const DevScene &S = P.s;
        const uint64_t path = (uint64_t)(P.path0 + slot);
        const float3 o = f4xyz(o4), d = f4xyz(d4);
        const float t = hv.x;
        const int code = __float_as_int(hv.y);
        const unsigned fl = flags_of(o4.w);
        const bool le = (fl & PFL_LE) != 0, inobj = (fl & PFL_IN) != 0;
        const float4 beta4 = P.beta_q[cur][i];
        beta = f4xyz(beta4);
        const bool last = bounce + 1 >= P.max_depth;
        float3 addL = mk3(0, 0, 0);
        if (t > 0.0f) {
            const int id = code & 0x7fffffff;
            const DevMaterial m = S.materials[prim_material(S, id)];
            const float3 p = rn_madd(o, d, t);
            const float3 nrm = surface_normal(S, id, code < 0, hv.z, hv.w, o, p, m);
            if (inobj) {  // BeerLambertLaw over the segment the previous vertex sent inside
                const float3 a = S.materials[__float_as_int(beta4.w)].rgb;
                beta = beta * mk3(expf(-a.x * t), expf(-a.y * t), expf(-a.z * t));
            }
            // Texture::Pattern scales what this vertex returns (raytracer.cpp:69-70)
            if (S.prim_tex) beta = beta * tex_pattern(S, id, p);
            const float3 wo = -d;
            const Uniform4 U0 = path_uniforms(path, bounce, 0, P.k0, P.k1);
            if (m.type == MAT_SPECULAR) {
                nx_d = mirror_dir(wo, nrm);
                float3 albedo = m.rgb;
                if (id < S.n_tris && S.tri_albedo) albedo = f4xyz(__ldg(&S.tri_albedo[id]));
                beta = beta * (albedo * m.kd);
                nx_o = p;
                nx_flags = PFL_LE;
                want_next = !last;
            } else if (m.type == MAT_DIELECTRIC) {
                const float kr = fresnel_kr(d, nrm, m.eta_in, m.eta_out);
                const float kt = 1.0f - kr;
                float c;
                bool entering;
                if (kr != 0.0f && U0.u[0] <= kr) {
                    nx_d = fresnel_reflect_dir(wo, nrm, c);
                    entering = c < 0.0f;
                    beta = beta * (kr * (1.0f / kr));
                } else {
                    nx_d = refract_dir(wo, nrm, m.eta_in, m.eta_out, c);
                    entering = c > 0.0f;
                    const float eta = inobj ? m.eta_in / m.eta_out : m.eta_out / m.eta_in;
                    beta = beta * (1.0f / (eta * eta) * kt * (1.0f / kt));
                }
                nx_o = p;
                nx_flags = PFL_LE | (entering ? PFL_IN : 0);
                enter_mat = prim_material(S, id);
                want_next = !last;
            } else if (m.type == MAT_EMISSIVE) {
                if (le && !inobj && -dot3(d, nrm) > 0.0f) addL = beta * m.le;
            } else if (S.n_lights > 0 && (m.type == MAT_MATTE || (m.type == MAT_GLOSSY && m.kd != 0.0f &&
                                                                  1.0f <= m.kd_pdf))) {
                const Uniform4 U1 = path_uniforms(path, bounce, 1, P.k0, P.k1);
                const LightSample ls = sample_light(S, U0.u[3], U1.u[0], U1.u[1], p, nrm);
                float3 wi;
                float dist, G;
                if (nee_setup(ls, p, wi, dist, G)) {
                    float3 albedo = m.rgb;
                    if (id < S.n_tris && S.tri_albedo) albedo = f4xyz(__ldg(&S.tri_albedo[id]));
                    const float3 f = albedo * RUMI_INV_PI_F * m.kd;
                    const float cost = fmaxf(dot3(wi, nrm), 0.0f);
                    float3 direct = f * ls.Li * cost * G / ls.pdf;
                    if (m.type == MAT_GLOSSY) direct = direct * (1.0f / m.kd_pdf);
                    float tr = 1.0f;
                    if (S.volume.present) {
                        const Uniform4 U2 = path_uniforms(path, bounce, 2, P.k0, P.k1);
                        float smax_sh = 0.0f;
                        tr = volume_shadow_tr(S.volume, p, wi, dist, U2.u[2], &smax_sh);
                    }
                    const float3 c = beta * direct;  // zero contributions are not traced
                    if (tr > 0.0f && (c.x != 0.0f || c.y != 0.0f || c.z != 0.0f)) {
                        want_sh = true;
                        sh_o = p;
                        sh_d = wi;
                        sh_tmax = dist;
                        sh_c = c;
                    }
                }
            }
        }
        if (addL.x != 0.0f || addL.y != 0.0f || addL.z != 0.0f) {
            float4 l = P.L[slot];
            l.x += addL.x; l.y += addL.y; l.z += addL.z;
            P.L[slot] = l;
        }
    }
    int kn, ks;
    block_push2(&P.cnt[nxt], want_next, kn, shadow_count(P), want_sh, ks);
    if (want_next) {
        store_ray(P.ray[nxt], kn, make_float4(nx_o.x, nx_o.y, nx_o.z, pack_slot(slot, nx_flags)),
                  make_float4(nx_d.x, nx_d.y, nx_d.z, FLT_MAX));
        P.beta_q[nxt][kn] = make_float4(beta.x, beta.y, beta.z, __int_as_float(enter_mat));
    }
    if (want_sh) {
        store_ray(P.sh_ray, ks, make_float4(sh_o.x, sh_o.y, sh_o.z, __int_as_float(slot)),
                  make_float4(sh_d.x, sh_d.y, sh_d.z, sh_tmax));
        P.sh_c[ks] = make_float4(sh_c.x, sh_c.y, sh_c.z, 0.0f);
    }
}

// One warp per pixel: the pixel's samples are summed in sample order by lane 0 after
// a coalesced load of up to 32 samples at a time.
__global__ void pt_resolve(PtLaunch P) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= P.n_pix) return;
    float3 acc = mk3(0.0f, 0.0f, 0.0f);
    int nan = 0;
    const long long gp = (long long)P.pix0 + warp;
    int spp = P.spp;
    size_t base = (size_t)warp * P.spp;
    if (P.scenes) {
        const int k = find_scene(P.scene_pix0, P.n_scenes, gp);
        spp = P.scene_spp[k];
        base = (size_t)(P.scene_path0[k] + (gp - P.scene_pix0[k]) * spp - P.path0);
    }
    for (int s0 = 0; s0 < spp; s0 += 32) {
        const int s = s0 + lane;
        float4 l = make_float4(0, 0, 0, 0);
        if (s < spp) l = P.L[base + s];
        const int cnt = min(32, spp - s0);
        for (int k = 0; k < cnt; ++k) {
            const float x = __shfl_sync(0xffffffffu, l.x, k);
            const float y = __shfl_sync(0xffffffffu, l.y, k);
            const float z = __shfl_sync(0xffffffffu, l.z, k);
            if (x != x || y != y || z != z)
                ++nan;
            else {
                acc.x += x; acc.y += y; acc.z += z;
            }
        }
    }
    if (lane == 0) {
        const size_t px = (size_t)gp * 3;
        P.film[px + 0] = acc.z;  // B
        P.film[px + 1] = acc.y;  // G
        P.film[px + 2] = acc.x;  // R
        if (nan) atomicAdd(&P.stats[S_NAN], (unsigned long long)nan);
    }
}

static inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }
static inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Traversal scheme index (traverse_queue MODE) from rumi_render_params.trace_mode:
// 1..5 select modes 0..4, 0 selects the default, the speculative while-while walk over the
// four-wide tree, the fastest on the BVH-bound workload.
static inline int trace_scheme(int trace_mode) {
    return trace_mode >= 1 && trace_mode <= 5 ? trace_mode - 1 : DEFAULT_WALK_MODE;
}
// The scheme of a scene's frames: the default walk gives way to testing the records in step
// (SCHEME_FEW) where the four-wide tree is a single node of few records, unless the call asks for a
// scheme or for traversal counts.  Closest-hit / any-hit ms of a 512x512, 16 spp, depth-6 frame,
// walk against that: 10 triangles and a light (7 records) 0.71 / 0.55 and 0.68 / 0.54; 12
// triangles, a light and a sphere (9) 0.96 / 0.61 and 0.93 / 0.65; and of the 256x256, 16 spp,
// depth-8 Cornell frame (9 records) 0.31 / 0.23 and 0.27 / 0.22.  Whole frames: one-node scenes of 7 and 8
// records 0.60 / 0.63 walked and 0.51 / 0.54 in step, the box with 2, 4, 6 and 8 more triangles (8 to 11
// records) 0.84 / 0.85 / 0.90 / 0.91 and 0.78 / 0.80 / 0.82 / 0.87; no scene with more records came out as
// one node.
static inline int scene_scheme(const rumi_scene *sc, const rumi_render_params *p) {
    const bool few = sc->n_wide == 1 && sc->n_recs <= RUMI_FEW_RECORDS;
    return few && DEFAULT_WALK_MODE == SCHEME_WIDE && p->trace_mode == 0 && !(p->flags & RUMI_FLAG_STATS)
               ? SCHEME_FEW
               : trace_scheme(p->trace_mode);
}
bool uses_bvh8(int trace_mode) { return trace_scheme(trace_mode) == SCHEME_EIGHT; }

using ExtendKernel = void (*)(PtLaunch, int);
using ShadowKernel = void (*)(PtLaunch);

// Shared-memory stack depth from rumi_render_params.stack_depth: 8, 16 or 32 entries per
// thread (0 = 16).  Only the while-while walks (SCHEME_WIDE, SCHEME_EIGHT) come in all three depths.
// Measured on the 1024x1024x64 BVH-bound frame (four-wide walk, closest-hit / any-hit ms):
// 8: 65.8 / 35.9, 16: 65.7 / 35.2, 32 with the L1 carveout sized to it: 65.5 / 35.2 (before
// the rays were ordered).
static inline int stack_entries(int stack_depth) { return stack_depth == 8 || stack_depth == 32 ? stack_depth : 16; }

// Kernel selection and launches.  A host build of this file (RUMI_HOST_BUILD: the kernels
// compiled as plain C++ for the CPU tests) leaves them out; it keeps the wave layout below.
#ifndef RUMI_HOST_BUILD
template <bool STATS>
static ExtendKernel extend_kernel(int mode, int smem) {
    switch (mode) {
        case SCHEME_BATCH: return pt_extend<SCHEME_BATCH, STATS>;
        case SCHEME_REFILL: return pt_extend<SCHEME_REFILL, STATS>;
        case SCHEME_LEAVES: return pt_extend<SCHEME_LEAVES, STATS>;
        case SCHEME_FEW: return pt_extend<SCHEME_FEW, STATS, 1>;
        case SCHEME_WIDE:
            return smem == 8    ? pt_extend<SCHEME_WIDE, STATS, 8>
                   : smem == 16 ? pt_extend<SCHEME_WIDE, STATS, 16>
                                : pt_extend<SCHEME_WIDE, STATS>;
        default:
            return smem == 8    ? pt_extend<SCHEME_EIGHT, STATS, 8>
                   : smem == 16 ? pt_extend<SCHEME_EIGHT, STATS, 16>
                                : pt_extend<SCHEME_EIGHT, STATS>;
    }
}

template <bool ADJ>
static ShadowKernel shadow_kernel(int mode, int smem) {
    switch (mode) {
        case SCHEME_BATCH: return pt_shadow<SCHEME_BATCH, ADJ>;
        case SCHEME_REFILL: return pt_shadow<SCHEME_REFILL, ADJ>;
        case SCHEME_LEAVES: return pt_shadow<SCHEME_LEAVES, ADJ>;
        case SCHEME_FEW: return pt_shadow<SCHEME_FEW, ADJ, 1>;
        case SCHEME_WIDE:
            return smem == 8    ? pt_shadow<SCHEME_WIDE, ADJ, 8>
                   : smem == 16 ? pt_shadow<SCHEME_WIDE, ADJ, 16>
                                : pt_shadow<SCHEME_WIDE, ADJ>;
        default:
            return smem == 8    ? pt_shadow<SCHEME_EIGHT, ADJ, 8>
                   : smem == 16 ? pt_shadow<SCHEME_EIGHT, ADJ, 16>
                                : pt_shadow<SCHEME_EIGHT, ADJ>;
    }
}

// How a bounce's shading leaves the next rays.  order: the wave's rays are ordered.  The general kernel
// gains nothing from grouping where the records are tested in step and goes without it; the lean one is
// the other way round (0.40 against 0.38 ms, Cornell frame).
static Group shade_group(bool lean, int mode, bool order) {
    return order ? GROUP_FRAME : lean || mode != SCHEME_FEW ? GROUP_BLOCK : GROUP_NONE;
}

// Forward shading of one bounce.  lean: the instantiation without the medium, texture,
// image-based-light and subsurface branches, for scenes that have none of them; it and the general
// one differ in the compiler's FMA contraction, not in the algorithm, so every forward pass of a scene
// (render, forward with or without kept radiance, the first pass of backward, a batch that is lean as
// the scene is) takes the same of the two.  Their instantiations by group share the text of a path's
// arithmetic but are compiled one by one: that frames of one scene are the same bits with either is
// tested (over textures, image-based light, subsurface and media), not guaranteed by construction.
static void launch_shade(bool lean, Group group, cudaStream_t st, const PtLaunch &L, int b) {
    const auto k = lean ? (group == GROUP_FRAME ? pt_shade<false, true, GROUP_FRAME> : pt_shade<false, true, GROUP_BLOCK>)
                        : (group == GROUP_FRAME   ? pt_shade<false, false, GROUP_FRAME>
                           : group == GROUP_BLOCK ? pt_shade<false, false, GROUP_BLOCK>
                                                  : pt_shade<false, false, GROUP_NONE>);
    k<<<cdiv(L.n_paths, SHADE_THREADS), SHADE_THREADS, 0, st>>>(L, b);
}

template <bool STATS>
static void launch_extend(int mode, int smem, int grid, cudaStream_t st, const PtLaunch &L, int b) {
    extend_kernel<STATS>(mode, smem)<<<grid, TRACE_THREADS, 0, st>>>(L, b);
}

template <bool ADJ>
static void launch_shadow(int mode, int smem, int grid, cudaStream_t st, const PtLaunch &L) {
    shadow_kernel<ADJ>(mode, smem)<<<grid, TRACE_THREADS, 0, st>>>(L);
}

// Resident blocks per SM of a persistent traversal kernel, asked of the runtime once per kernel
// and device (about 2 us a question, as long as a small frame's launch).  The first question
// also sets the kernel's shared-memory preference to just what `blocks` resident blocks need, so
// that the rest of the unified L1 / shared storage stays L1.
static int resident_blocks(const void *k, int blocks) {
    static std::mutex mutex;
    static std::map<std::pair<const void *, int>, int> known;
    int device = 0;
    cudaGetDevice(&device);
    std::lock_guard<std::mutex> lock(mutex);
    const auto it = known.find({k, device});
    if (it != known.end()) return it->second;
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k) == cudaSuccess) {
        const int need = blocks * ((int)fa.sharedSizeBytes + 1024);  // 1 KB per block is the runtime's
        const int pct = (need * 100 + 228 * 1024 - 1) / (228 * 1024);
        cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, pct > 100 ? 100 : pct);
    }
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, TRACE_THREADS, 0) != cudaSuccess || occ < 1) return 1;
    known[{k, device}] = occ;
    return occ;
}

// Persistent grid of a traversal kernel for at most n rays: blocks per SM at the kernel's
// occupancy (capped by blocks_per_sm > 0), and no block that could not get a ray.
template <typename K>
static int trace_grid(K k, int min_blocks, int num_sms, int blocks_per_sm, long long n) {
    int occ = resident_blocks((const void *)k, min_blocks);
    if (blocks_per_sm > 0 && blocks_per_sm < occ) occ = blocks_per_sm;
    const long long useful = (n + TRACE_THREADS - 1) / TRACE_THREADS, all = (long long)num_sms * occ;
    return (int)(useful < 1 ? 1 : (useful < all ? useful : all));
}

static void trace_grids(int mode, int smem, int num_sms, int blocks_per_sm, bool adj, bool stats, long long n, int &grid,
                        int &grid_sh) {
    grid = trace_grid(stats ? extend_kernel<true>(mode, smem) : extend_kernel<false>(mode, smem),
                      trace_min_blocks(mode, true), num_sms, blocks_per_sm, n);
    grid_sh = trace_grid(adj ? shadow_kernel<true>(mode, smem) : shadow_kernel<false>(mode, smem),
                         trace_min_blocks(mode, false), num_sms, blocks_per_sm, n);
}

#endif  // RUMI_HOST_BUILD

// Carves the wave state for Wp paths out of ws (pt_workspace_bytes(Wp) bytes) and clears
// every optional field; returns the first byte after it.
static char *carve_wave(PtLaunch &L, void *ws, size_t Wp) {
    memset(&L, 0, sizeof(L));
    const size_t f4 = align256(Wp * sizeof(float4));
    char *w = (char *)ws;
    L.ray[0] = (float4 *)w; w += 2 * f4;
    L.ray[1] = (float4 *)w; w += 2 * f4;
    L.hit = (float4 *)w; w += f4;
    L.sh_ray = (float4 *)w; w += 2 * f4;
    L.sh_c = (float4 *)w; w += f4;
    L.beta_q[0] = (float4 *)w; w += f4;
    L.beta_q[1] = (float4 *)w; w += f4;
    L.L = (float4 *)w; w += f4;
    L.cnt = (int *)w; w += align256(C_NUM * sizeof(int));
    L.stats = (unsigned long long *)w; w += align256(S_NUM * sizeof(unsigned long long));
    return w;
}

// Device bytes of the wave state for `paths` paths in flight (queues, path state,
// counters): 176 bytes per path plus alignment and counters.
size_t pt_workspace_bytes(long long paths) {
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t Wp = (size_t)paths;
    return 11 * al(Wp * sizeof(float4)) + al(C_NUM * sizeof(int)) + al(S_NUM * sizeof(unsigned long long));
}

#ifndef RUMI_HOST_BUILD
// Counters and statistics (adjacent in the wave state) to zero.
static void clear_counters(const PtLaunch &L, cudaStream_t stream) {
    cudaMemsetAsync(L.cnt, 0, align256(C_NUM * sizeof(int)) + S_NUM * sizeof(unsigned long long), stream);
}

// The scene's second stream and its fork / join events, made on first use.
static rumi_status ensure_aux(rumi_scene *sc) {
    if (sc->aux_stream) return RUMI_OK;
    cudaError_t e = cudaStreamCreateWithFlags(&sc->aux_stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sc->ev_fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&sc->ev_join, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_status(e, "auxiliary stream");
    return RUMI_OK;
}

// Device bytes for ordering the rays of a wave, after its wave state.
static size_t sort_bytes(long long paths) {
    return 2 * SORT_BINS * sizeof(int) + align256((size_t)paths * sizeof(int2)) + (size_t)paths * sizeof(int);
}
// Whether a frame's waves have their rays ordered: enough rays that several share a bin, and a tree
// whose walk is worth more than the ordering.  Depth-10 frames of a displaced sphere in a box, in
// order against as they come, 1, 2, 4, 8 and 17 million paths: of a million triangles 3.34 / 3.12,
// 5.04 / 4.97, 8.32 / 8.70, 15.2 / 16.2, 27.8 / 30.8 ms; of 1034 triangles 1.86 / 1.71,
// 3.05 / 2.96, 5.22 / 5.31, 9.66 / 10.2, 18.1 / 19.5 ms.  Of 266 triangles (under the line of
// nodes) 4.47 / 4.44 at 4 million and 15.8 / 16.4 at 17; of 26 triangles 13.2 / 12.9 at 17.
static bool sort_wave(const rumi_scene *sc, const rumi_render_params *p, long long paths) {
    return p->integrator == RUMI_PATH_TRACER && scene_scheme(sc, p) == SCHEME_WIDE && paths >= RUMI_SORT_PATHS &&
           sc->n_wide >= RUMI_SORT_NODES;
}

rumi_status pt_render(rumi_scene *sc, const rumi_render_params *p, float *film_dev, rumi_render_stats *stats,
                      cudaStream_t stream, float4 *keep_L) {
    const long long total_pix = (long long)sc->dev.width * sc->dev.height;
    long long wave = p->wave_paths > 0 ? p->wave_paths : RUMI_DEFAULT_WAVE_PATHS;
    long long pix_per_wave = wave / p->spp;
    if (pix_per_wave < 1) pix_per_wave = 1;
    if (pix_per_wave > total_pix) pix_per_wave = total_pix;
    const long long n_paths_max = pix_per_wave * p->spp;
    if (n_paths_max > 0x3fffffffLL) {  // slots are 30-bit (pack_slot)
        set_error("wave_paths too large");
        return RUMI_ERR_INVALID_ARG;
    }
    const size_t bytes = pt_workspace_bytes(n_paths_max);
    // without memory for ordering the rays the frame goes without the order
    const bool sort = sort_wave(sc, p, n_paths_max) && try_workspace(sc, bytes + sort_bytes(n_paths_max));
    rumi_status st = ensure_workspace(sc, bytes);
    if (st != RUMI_OK) return st;
    if (uses_bvh8(p->trace_mode) && (st = ensure_bvh8(sc)) != RUMI_OK) return st;
    if ((st = ensure_aux(sc)) != RUMI_OK) return st;
    return pt_render_in(sc, p, film_dev, stats, stream, sc->ws, pix_per_wave,
                        RUMI_PT_OVERLAP != 0 && !(p->flags & RUMI_FLAG_SERIAL), keep_L, sort);
}

// The frame loop over waves of pix_per_wave pixels, with the wave state carved out of
// `ws` (pt_workspace_bytes(pix_per_wave * spp) bytes).
rumi_status pt_render_in(rumi_scene *sc, const rumi_render_params *p, float *film_dev, rumi_render_stats *stats,
                         cudaStream_t stream, void *ws, long long pix_per_wave, bool overlap, float4 *keep_L,
                         bool sort) {
    const int W = sc->dev.width, H = sc->dev.height;
    const int spp = p->spp;
    const long long total_pix = (long long)W * H;
    const size_t Wp = (size_t)(pix_per_wave * spp);
    PtLaunch L;
    carve_wave(L, ws, Wp);
    L.s = sc->dev;
    L.spp = spp;
    // RayTracer::Trace shades trace depths 0..max_depth (raytracer.cpp:41-42)
    const bool whitted = p->integrator == RUMI_RAY_TRACER;
    const int bounces = whitted ? p->max_depth + 1 : p->max_depth;
    L.max_depth = bounces;
    L.k0 = (uint32_t)p->seed;
    L.k1 = (uint32_t)(p->seed >> 32) ^ 0x5851F42Du;
    int d = 0;
    while ((d + 1) * (d + 1) <= spp) ++d;
    L.grid_d = d;
    L.square = d * d == spp;
    L.film = film_dev;
    clear_counters(L, stream);

    // traversal scheme and persistent grid (autotuner knobs; 0 = defaults)
    const int mode = scene_scheme(sc, p);
    const int smem = stack_entries(p->stack_depth);
    L.refill_min = p->refill_min > 0 ? p->refill_min : 8;
    const bool timing = (p->flags & RUMI_FLAG_TIMING) != 0;
    const bool count_stats = (p->flags & RUMI_FLAG_STATS) != 0;
    int grid = 0, shadow_grid = 0;
    trace_grids(mode, smem, sc->num_sms, p->blocks_per_sm, false, count_stats, (long long)Wp, grid, shadow_grid);
    const bool lean = shade_lean(sc);
    const Group group = shade_group(lean, mode, sort);
    if (sort) {
        char *w = (char *)ws + pt_workspace_bytes((long long)Wp);
        L.sort_bins = (int *)w; w += SORT_BINS * sizeof(int);
        L.sort_base = (int *)w; w += SORT_BINS * sizeof(int);
        L.sort_key = (int2 *)w; w += align256(Wp * sizeof(int2));
        L.sort_perm = (int *)w;
        cudaMemsetAsync(L.sort_bins, 0, SORT_BINS * sizeof(int), stream);
    }
    // orders the rays that shading of bounce b has queued
    auto sort_next = [&](int b) {
        L.sorted = sort && b + 1 < bounces;
        if (!L.sorted) return;
        const int queue = (b & 1) ^ 1, blocks = cdiv(L.n_paths, 256), resident = sc->num_sms * 32;
        pt_sort_bases<<<SORT_BINS / (4 * SORT_THREADS), SORT_THREADS, 0, stream>>>(L, queue);
        pt_sort_order<<<blocks < resident ? blocks : resident, 256, 0, stream>>>(L, queue);
    };
    std::vector<cudaEvent_t> evs;
    auto mark_on = [&](cudaStream_t st_) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        cudaEventRecord(e, st_);
        evs.push_back(e);
    };
    auto mark = [&]() { mark_on(stream); };
    // event indices of (begin, end) per launch kind
    std::vector<std::pair<int, int>> ext_ev, shade_ev, sh_ev;
    if (timing) mark();
    long long waves = 0;
    for (long long pix0 = 0; pix0 < total_pix; pix0 += pix_per_wave) {
        const long long n_pix = pix0 + pix_per_wave <= total_pix ? pix_per_wave : total_pix - pix0;
        L.pix0 = (int)pix0;
        L.n_pix = (int)n_pix;
        L.n_paths = (int)(n_pix * spp);
        L.path0 = pix0 * spp;
        pt_generate<<<cdiv(L.n_paths, 256), 256, 0, stream>>>(L);
        if (overlap) {
            // shadow rays of bounce b are traced on the auxiliary stream while bounce b + 1's
            // closest-hit rays are traced here: neither reads what the other writes (shadow
            // queue and per-path radiance vs ray queue and hits); shading of b + 1 waits
            // for both, as it refills the shadow queue and adds to the radiance
            // (with timing, a closest-hit launch's events include the time it shares the
            // GPU with the previous bounce's any-hit launch)
            L.chained = 1;
            for (int b = 0; b < bounces; ++b) {
                L.sh_set = b & 1;
                int e0 = 0;
                if (timing) { e0 = (int)evs.size(); mark(); }
                if (count_stats)
                    launch_extend<true>(mode, smem, grid, stream, L, b);
                else
                    launch_extend<false>(mode, smem, grid, stream, L, b);
                if (timing) { mark(); ext_ev.push_back({e0, e0 + 1}); }
                if (b > 0) cudaStreamWaitEvent(stream, sc->ev_join, 0);
                if (timing) { e0 = (int)evs.size(); mark(); }
                if (whitted)
                    pt_shade_whitted<<<cdiv(L.n_paths, SHADE_THREADS), SHADE_THREADS, 0, stream>>>(L, b);
                else
                    launch_shade(lean, group, stream, L, b);
                if (timing) { mark(); shade_ev.push_back({e0, e0 + 1}); }
                const bool aside = b + 1 < bounces;
                cudaStream_t ss = aside ? sc->aux_stream : stream;
                if (aside) {
                    cudaEventRecord(sc->ev_fork, stream);
                    cudaStreamWaitEvent(sc->aux_stream, sc->ev_fork, 0);
                }
                if (timing) { e0 = (int)evs.size(); mark_on(ss); }
                launch_shadow<false>(mode, smem, shadow_grid, ss, L);
                if (timing) { mark_on(ss); sh_ev.push_back({e0, e0 + 1}); }
                if (aside) cudaEventRecord(sc->ev_join, sc->aux_stream);
                sort_next(b);
            }
            pt_resolve<<<cdiv(L.n_pix * 32LL, 256), 256, 0, stream>>>(L);
            if (keep_L)
                cudaMemcpyAsync(keep_L + L.path0, L.L, sizeof(float4) * (size_t)L.n_paths, cudaMemcpyDeviceToDevice,
                                stream);
            ++waves;
            continue;
        }
        for (int b = 0; b < bounces; ++b) {
            pt_reset<<<1, 1, 0, stream>>>(L, b);
            int e0 = 0;
            if (timing) { e0 = (int)evs.size(); mark(); }
            if (count_stats)
                launch_extend<true>(mode, smem, grid, stream, L, b);
            else
                launch_extend<false>(mode, smem, grid, stream, L, b);
            if (timing) { mark(); ext_ev.push_back({e0, e0 + 1}); }
            if (timing) { e0 = (int)evs.size(); mark(); }
            if (whitted)
                pt_shade_whitted<<<cdiv(L.n_paths, SHADE_THREADS), SHADE_THREADS, 0, stream>>>(L, b);
            else
                launch_shade(lean, group, stream, L, b);
            if (timing) { mark(); shade_ev.push_back({e0, e0 + 1}); }
            if (timing) { e0 = (int)evs.size(); mark(); }
            launch_shadow<false>(mode, smem, shadow_grid, stream, L);
            if (timing) { mark(); sh_ev.push_back({e0, e0 + 1}); }
            sort_next(b);
        }
        pt_finish<<<1, 1, 0, stream>>>(L);
        pt_resolve<<<cdiv(L.n_pix * 32LL, 256), 256, 0, stream>>>(L);
        if (keep_L)
            cudaMemcpyAsync(keep_L + L.path0, L.L, sizeof(float4) * (size_t)L.n_paths, cudaMemcpyDeviceToDevice,
                            stream);
        ++waves;
    }
    if (timing) mark();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_status(e, "pt_render launch");
    unsigned long long h_stats[S_NUM];
    cudaMemcpyAsync(h_stats, L.stats, sizeof(h_stats), cudaMemcpyDeviceToHost, stream);
    e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) {
        for (auto ev : evs) cudaEventDestroy(ev);
        return cuda_status(e, "pt_render");
    }
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->paths = total_pix * spp;
        stats->nan_samples = (int64_t)h_stats[S_NAN];
        stats->rays_extend = (int64_t)h_stats[S_RAYS_EXT];
        stats->rays_shadow = (int64_t)h_stats[S_RAYS_SH];
        stats->extend_node_fetches = (int64_t)(h_stats[S_NODES] / 2);  // 16-byte units -> 32-byte nodes
        stats->extend_prim_tests = (int64_t)h_stats[S_PRIMS];
        stats->extend_launches = (int64_t)waves * bounces;
        stats->shade_launches = stats->extend_launches;
        stats->shadow_launches = stats->extend_launches;
        if (timing) {
            float ms;
            for (auto &pr : ext_ev) { cudaEventElapsedTime(&ms, evs[pr.first], evs[pr.second]); stats->extend_ms += ms; }
            for (auto &pr : shade_ev) { cudaEventElapsedTime(&ms, evs[pr.first], evs[pr.second]); stats->shade_ms += ms; }
            for (auto &pr : sh_ev) { cudaEventElapsedTime(&ms, evs[pr.first], evs[pr.second]); stats->shadow_ms += ms; }
            cudaEventElapsedTime(&ms, evs.front(), evs.back());
            stats->total_ms = ms;
        }
    }
    for (auto ev : evs) cudaEventDestroy(ev);
    return RUMI_OK;
}

// ---------------------------------------------------------------- path-replay adjoint
// Device bytes of the adjoint's wave state: the rendering wave state plus, per path, the
// first pass's radiance, the loss weights and the shadow-ray scores.
size_t pt_adjoint_workspace_bytes(long long paths) {
    const size_t Wp = (size_t)paths;
    return pt_workspace_bytes(paths) + 2 * align256(Wp * sizeof(float4)) + align256(Wp * sizeof(float2));
}

// Gradients of <dfilm, film> for the frame rumi_render produces with the same parameters:
// g_albedo (n_tris * 3, RGB; may be null) and g_medium (GM_NUM; may be null) are
// overwritten.  Each wave is traced twice: pass 1 records every path's radiance, pass 2
// replays the same random numbers with the scores of pt_shade<true> / pt_shadow<0, true>.
rumi_status pt_backward(rumi_scene *sc, const rumi_render_params *p, const float *dfilm_dev, float *g_albedo,
                        float *g_medium, rumi_render_stats *stats, cudaStream_t stream) {
    const int W = sc->dev.width, H = sc->dev.height;
    const int spp = p->spp;
    const long long total_pix = (long long)W * H;
    long long wave = p->wave_paths > 0 ? p->wave_paths : RUMI_DEFAULT_WAVE_PATHS;
    long long pix_per_wave = wave / spp;
    if (pix_per_wave < 1) pix_per_wave = 1;
    if (pix_per_wave > total_pix) pix_per_wave = total_pix;
    const size_t Wp = (size_t)(pix_per_wave * spp);
    if (Wp > 0x3fffffffULL) {
        set_error("wave_paths too large");
        return RUMI_ERR_INVALID_ARG;
    }
    rumi_status st = ensure_workspace(sc, pt_adjoint_workspace_bytes((long long)Wp));
    if (st != RUMI_OK) return st;
    if (uses_bvh8(p->trace_mode) && (st = ensure_bvh8(sc)) != RUMI_OK) return st;
    const bool overlap = RUMI_PT_OVERLAP != 0 && !(p->flags & RUMI_FLAG_SERIAL);
    if (overlap && (st = ensure_aux(sc)) != RUMI_OK) return st;
    // the forward pass of this very frame kept its per-path radiance: pass 1 is not traced
    const bool reuse = sc->kept_valid && sc->kept_seed == p->seed && sc->kept_spp == spp &&
                       sc->kept_depth == p->max_depth && sc->kept_cap >= total_pix * spp;
    float *gm_scratch = nullptr;
    cudaError_t e = cudaSuccess;
    if (!g_medium) {
        e = dalloc((void **)&gm_scratch, GM_NUM * sizeof(float), stream);
        if (e != cudaSuccess) return cuda_status(e, "adjoint scratch");
        g_medium = gm_scratch;
    }
    PtLaunch A;
    char *w = carve_wave(A, sc->ws, Wp);
    A.s = sc->dev;
    A.spp = spp;
    A.max_depth = p->max_depth;
    A.k0 = (uint32_t)p->seed;
    A.k1 = (uint32_t)(p->seed >> 32) ^ 0x5851F42Du;
    int d = 0;
    while ((d + 1) * (d + 1) <= spp) ++d;
    A.grid_d = d;
    A.square = d * d == spp;
    A.refill_min = 8;
    A.chained = 1;
    PtLaunch B = A;
    float4 *Lt = (float4 *)w; w += align256(Wp * sizeof(float4));
    B.Lt = Lt;
    B.dls = (float4 *)w; w += align256(Wp * sizeof(float4));
    B.sh_s = (float2 *)w;
    B.dfilm = dfilm_dev;
    B.g_albedo = g_albedo;
    B.g_medium = g_medium;
    clear_counters(A, stream);
    cudaMemsetAsync(g_medium, 0, GM_NUM * sizeof(float), stream);
    if (g_albedo) cudaMemsetAsync(g_albedo, 0, sizeof(float) * 3 * (size_t)sc->dev.n_tris, stream);

    // the same traversal scheme as rumi_render, so both passes and the forward frame
    // resolve exact-distance ties alike
    const int mode = scene_scheme(sc, p);
    const bool lean = shade_lean(sc);
    const int smem = stack_entries(p->stack_depth);
    A.refill_min = B.refill_min = p->refill_min > 0 ? p->refill_min : 8;
    int grid = 0, grid_sh = 0, grid_dummy = 0, grid_sh_adj = 0;
    trace_grids(mode, smem, sc->num_sms, p->blocks_per_sm, false, false, (long long)Wp, grid, grid_sh);
    trace_grids(mode, smem, sc->num_sms, p->blocks_per_sm, true, false, (long long)Wp, grid_dummy, grid_sh_adj);

    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (p->flags & RUMI_FLAG_TIMING) {
        cudaEventCreate(&e0);
        cudaEventCreate(&e1);
        cudaEventRecord(e0, stream);
    }
    long long waves = 0;
    for (long long pix0 = 0; pix0 < total_pix; pix0 += pix_per_wave) {
        const long long n_pix = pix0 + pix_per_wave <= total_pix ? pix_per_wave : total_pix - pix0;
        for (PtLaunch *L : {&A, &B}) {
            L->pix0 = (int)pix0;
            L->n_pix = (int)n_pix;
            L->n_paths = (int)(n_pix * spp);
            L->path0 = pix0 * spp;
        }
        // both passes on the two-stream schedule of pt_render_in: each bounce's shadow rays
        // beside the next bounce's closest-hit rays, shading after both
        auto pass = [&](PtLaunch &X, bool adj) {
            pt_generate<<<cdiv(X.n_paths, 256), 256, 0, stream>>>(X);
            for (int b = 0; b < p->max_depth; ++b) {
                X.sh_set = b & 1;
                launch_extend<false>(mode, smem, grid, stream, X, b);
                if (b > 0 && overlap) cudaStreamWaitEvent(stream, sc->ev_join, 0);
                if (adj)
                    pt_shade<true><<<cdiv(X.n_paths, SHADE_THREADS), SHADE_THREADS, 0, stream>>>(X, b);
                else
                    launch_shade(lean, shade_group(lean, mode, false), stream, X, b);
                const bool aside = overlap && b + 1 < p->max_depth;
                cudaStream_t ss = aside ? sc->aux_stream : stream;
                if (aside) {
                    cudaEventRecord(sc->ev_fork, stream);
                    cudaStreamWaitEvent(sc->aux_stream, sc->ev_fork, 0);
                }
                if (adj)
                    launch_shadow<true>(mode, smem, grid_sh_adj, ss, X);
                else
                    launch_shadow<false>(mode, smem, grid_sh, ss, X);
                if (aside) cudaEventRecord(sc->ev_join, sc->aux_stream);
            }
        };
        // pass 1: radiance of every path (or the radiance rumi_forward kept for this frame)
        if (reuse) {
            cudaMemcpyAsync(Lt, sc->kept_L + A.path0, sizeof(float4) * (size_t)A.n_paths, cudaMemcpyDeviceToDevice,
                            stream);
        } else {
            pass(A, false);
            cudaMemcpyAsync(Lt, A.L, sizeof(float4) * (size_t)A.n_paths, cudaMemcpyDeviceToDevice, stream);
        }
        // pass 2: replay with the scores
        pass(B, true);
        ++waves;
    }
    if (e1) cudaEventRecord(e1, stream);
    e = cudaGetLastError();
    unsigned long long h_stats[S_NUM];
    if (e == cudaSuccess) e = cudaMemcpyAsync(h_stats, A.stats, sizeof(h_stats), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    dfree(gm_scratch, stream);
    if (e != cudaSuccess) {
        if (e0) cudaEventDestroy(e0);
        if (e1) cudaEventDestroy(e1);
        return cuda_status(e, "pt_backward");
    }
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->paths = total_pix * spp;
        stats->nan_samples = (int64_t)h_stats[S_NAN];
        stats->rays_extend = (int64_t)h_stats[S_RAYS_EXT];
        stats->rays_shadow = (int64_t)h_stats[S_RAYS_SH];
        stats->extend_launches = (reuse ? 1 : 2) * waves * p->max_depth;
        stats->shade_launches = stats->extend_launches;
        stats->shadow_launches = stats->extend_launches;
        if (e0) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, e0, e1);
            stats->total_ms = ms;
        }
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    return RUMI_OK;
}

// ---------------------------------------------------------------- scene batches
// Device bytes of a multi-scene wave: the single-scene wave state plus each slot's scene.
size_t pt_batch_workspace_bytes(long long wave_paths) {
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    return pt_workspace_bytes(wave_paths) + al((size_t)wave_paths * sizeof(int));
}

// Enqueues one frame of a multi-scene batch without synchronising, so the sequence can
// be captured into a CUDA graph: waves over the batch's global pixel / path index space,
// every stage serving all scenes from shared queues.
rumi_status pt_enqueue_batch(const BatchFrame &F, void *ws, float *films, cudaStream_t stream, int num_sms,
                             cudaStream_t aux, cudaEvent_t ev_fork, cudaEvent_t ev_join) {
    PtLaunch L;
    L.slot_scene = (int *)carve_wave(L, ws, (size_t)F.wave_paths);
    L.max_depth = F.max_depth;
    L.film = films;
    L.scenes = F.scenes;
    L.scene_path0 = F.scene_path0;
    L.scene_pix0 = F.scene_pix0;
    L.scene_key = F.scene_key;
    L.scene_spp = F.scene_spp;
    L.n_scenes = F.n_scenes;
    L.spp = 1;
    L.refill_min = 8;
    L.chained = 1;
    clear_counters(L, stream);
    const int mb = trace_min_blocks(DEFAULT_WALK_MODE, true), mb_sh = trace_min_blocks(DEFAULT_WALK_MODE, false);
    for (const BatchWave &wv : F.waves) {
        L.pix0 = (int)wv.pix0;
        L.n_pix = (int)(wv.pix1 - wv.pix0);
        L.path0 = wv.path0;
        L.n_paths = (int)(wv.path1 - wv.path0);
        const int grid = trace_grid(pt_trace_multi<false>, mb, num_sms, F.blocks_per_sm, L.n_paths);
        const int grid_sh = trace_grid(pt_trace_multi<true>, mb_sh, num_sms, F.blocks_per_sm, L.n_paths);
        pt_generate<<<cdiv(L.n_paths, 256), 256, 0, stream>>>(L);
        // the two-stream schedule of pt_render_in (a graph capture takes the auxiliary
        // stream in through the fork event and every fork is joined before shading)
        for (int b = 0; b < F.max_depth; ++b) {
            L.sh_set = b & 1;
            pt_trace_multi<false><<<grid, TRACE_THREADS, 0, stream>>>(L, b);
            if (b > 0 && aux) cudaStreamWaitEvent(stream, ev_join, 0);
            launch_shade(F.lean, shade_group(F.lean, DEFAULT_WALK_MODE, false), stream, L, b);
            const bool aside = aux && b + 1 < F.max_depth;
            if (aside) {
                cudaEventRecord(ev_fork, stream);
                cudaStreamWaitEvent(aux, ev_fork, 0);
            }
            pt_trace_multi<true><<<grid_sh, TRACE_THREADS, 0, aside ? aux : stream>>>(L, b);
            if (aside) cudaEventRecord(ev_join, aux);
        }
        pt_resolve<<<cdiv(L.n_pix * 32LL, 256), 256, 0, stream>>>(L);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_status(e, "batch launch");
    return RUMI_OK;
}

// Device address of the 64-bit statistics inside a batch workspace.
unsigned long long *pt_batch_stats_ptr(void *ws, long long wave_paths) {
    PtLaunch L;
    carve_wave(L, ws, (size_t)wave_paths);  // the same layout pt_enqueue_batch carves
    return L.stats;
}

// ---------------------------------------------------------------- ray batches
struct TraceLaunch {
    DevScene s;
    const float4 *rays;  // 2 float4 per ray: (o, in_object), (d, tmax)
    float *t;
    int32_t *prim;
    long long n;
    int anyhit;
    unsigned long long *counters;  // [0] fetch, [1] nodes, [2] prims
};

// Ray queries: the renderer's default traversal scheme (speculative while-while with
// per-lane refill) over a caller's ray array, in chunks of at most 2^30 rays.
template <int MODE, bool ANYHIT, bool STATS>
__global__ void __launch_bounds__(TRACE_THREADS, trace_min_blocks(MODE, !ANYHIT))
    trace_batch_kernel(TraceLaunch T, long long first, int n, int *fetch_counter) {
    constexpr int SMEM = MODE == SCHEME_WIDE ? WALK_SMEM : STACK_SMEM;
    __shared__ int stack[SMEM * TRACE_THREADS];
    TraceStats st{0, 0};
    auto fetch = [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
        const long long k = first + i;
        const float4 o4 = T.rays[2 * k], d4 = T.rays[2 * k + 1];
        o = f4xyz(o4);
        d = f4xyz(d4);
        tmax = d4.w;
        in_obj = o4.w != 0.0f;
    };
    auto finish = [&](int i, const HitRec &h) {
        const long long k = first + i;
        T.t[k] = h.t;
        T.prim[k] = ANYHIT ? (h.t > 0.0f ? 1 : 0) : (h.t > 0.0f ? h.id : -1);
    };
    traverse_queue<MODE, ANYHIT, SMEM, STATS>(T.s, n, fetch_counter, 8, stack, fetch, finish, st);
    if (STATS) {
        atomicAdd(&T.counters[1], (unsigned long long)st.nodes);
        atomicAdd(&T.counters[2], (unsigned long long)st.prims);
    }
}

template <bool ANYHIT, bool STATS, int MODE = DEFAULT_WALK_MODE>
static void launch_trace_batch(const TraceLaunch &T, int num_sms, cudaStream_t stream) {
    const long long chunk = 1LL << 30;
    int k = 0;
    for (long long first = 0; first < T.n; first += chunk, ++k) {
        const int n = (int)(T.n - first < chunk ? T.n - first : chunk);
        // one fetch counter per chunk (counters[3 + k]; chunk count is bounded by the caller's n)
        int *ctr = reinterpret_cast<int *>(T.counters + 3) + k;
        const int grid = trace_grid(trace_batch_kernel<MODE, ANYHIT, STATS>, trace_min_blocks(MODE, !ANYHIT), num_sms, 0, n);
        trace_batch_kernel<MODE, ANYHIT, STATS><<<grid, TRACE_THREADS, 0, stream>>>(T, first, n, ctr);
    }
}

rumi_status trace_rays(rumi_scene *sc, int64_t n, const float *rays_dev, int anyhit, float *t_dev, int32_t *prim_dev,
                       int64_t *node_visits, int64_t *prim_tests, cudaStream_t stream) {
    const long long chunks = (n + (1LL << 30) - 1) >> 30;
    if (chunks > 64) {
        set_error("trace_rays: at most 2^36 rays per call");
        return RUMI_ERR_INVALID_ARG;
    }
    rumi_status st = ensure_workspace(sc, 256 + 3 * sizeof(unsigned long long) + 64 * sizeof(int));
    if (st != RUMI_OK) return st;
    TraceLaunch T;
    T.s = sc->dev;
    T.rays = (const float4 *)rays_dev;
    T.t = t_dev;
    T.prim = prim_dev;
    T.n = n;
    T.anyhit = anyhit;
    T.counters = (unsigned long long *)sc->ws;
    cudaMemsetAsync(T.counters, 0, 3 * sizeof(unsigned long long) + 64 * sizeof(int), stream);
    const bool stats = node_visits != nullptr || prim_tests != nullptr;
    if (n > 0) {
        if (anyhit)
            stats ? launch_trace_batch<true, true>(T, sc->num_sms, stream)
                  : launch_trace_batch<true, false>(T, sc->num_sms, stream);
        else
            stats ? launch_trace_batch<false, true>(T, sc->num_sms, stream)
                  : launch_trace_batch<false, false>(T, sc->num_sms, stream);
    }
    unsigned long long h[3] = {0, 0, 0};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, T.counters, sizeof(h), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_status(e, "trace_rays");
    if (node_visits) *node_visits = (int64_t)(h[1] / 2);  // 16-byte units -> 32-byte nodes
    if (prim_tests) *prim_tests = (int64_t)h[2];
    return RUMI_OK;
}

static constexpr size_t STAGE_COUNTERS = 256 * 3;
static_assert(3 * sizeof(unsigned long long) + sizeof(int) <= STAGE_COUNTERS, "counters of one chunk");

bool make_stage(rumi_scene *sc) {
    return grow_optional(
        sc->stage, sc->stage_bytes, sc->stage_refused, (size_t)STAGED_RAYS * 40 + STAGE_COUNTERS,
        [](size_t n) {
            void *p = nullptr;
            if (cudaHostAlloc(&p, n, cudaHostAllocPortable) == cudaSuccess) return p;
            cudaGetLastError();
            return (void *)nullptr;
        },
        [](void *p) { cudaFreeHost(p); });
}

// A small query is all latency: three allocations, three pageable copies and three waits around
// a 10 us kernel.  Here the rays and zeroed counters go up in one page-locked copy and counters, t
// and prim come back in one, through memory the scene keeps (61 rays: 72 us before).
rumi_status trace_rays_staged(rumi_scene *sc, int64_t n, const float *rays, int anyhit, float *t, int32_t *prim,
                              int64_t *node_visits, int64_t *prim_tests, cudaStream_t stream) {
    constexpr size_t COUNTERS = STAGE_COUNTERS;
    const size_t b_rays = sizeof(float) * 8 * (size_t)n, b_t = sizeof(float) * (size_t)n, total = b_rays + COUNTERS + 2 * b_t;
    rumi_status st = ensure_workspace(sc, total);
    if (st != RUMI_OK) return st;
    char *dev = (char *)sc->ws, *host = (char *)sc->stage;
    memcpy(host, rays, b_rays);
    memset(host + b_rays, 0, COUNTERS);
    cudaMemcpyAsync(dev, host, b_rays + COUNTERS, cudaMemcpyHostToDevice, stream);
    TraceLaunch T;
    T.s = sc->dev;
    T.rays = (const float4 *)dev;
    T.counters = (unsigned long long *)(dev + b_rays);
    T.t = (float *)(dev + b_rays + COUNTERS);
    T.prim = (int32_t *)(dev + b_rays + COUNTERS + b_t);
    T.n = n;
    T.anyhit = anyhit;
    const bool stats = node_visits != nullptr || prim_tests != nullptr;
    if (anyhit)
        stats ? launch_trace_batch<true, true>(T, sc->num_sms, stream) : launch_trace_batch<true, false>(T, sc->num_sms, stream);
    else
        stats ? launch_trace_batch<false, true>(T, sc->num_sms, stream)
              : launch_trace_batch<false, false>(T, sc->num_sms, stream);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(host + b_rays, dev + b_rays, COUNTERS + 2 * b_t, cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_status(e, "trace_rays");
    unsigned long long h[3];
    memcpy(h, host + b_rays, sizeof(h));
    memcpy(t, host + b_rays + COUNTERS, b_t);
    memcpy(prim, host + b_rays + COUNTERS + b_t, b_t);
    if (node_visits) *node_visits = (int64_t)(h[1] / 2);  // 16-byte units -> 32-byte nodes
    if (prim_tests) *prim_tests = (int64_t)h[2];
    return RUMI_OK;
}

// Ray queries through the traversal scheme trace_mode selects (1..5, as rumi_render_params;
// 0 = the default), so a test can compare every scheme's hits on the same rays.
rumi_status trace_rays_scheme(rumi_scene *sc, int64_t n, const float *rays_dev, int anyhit, int trace_mode,
                              float *t_dev, int32_t *prim_dev, cudaStream_t stream) {
    if (n < 0 || n > (1LL << 30)) {
        set_error("trace_rays_scheme: 0 <= n <= 2^30");
        return RUMI_ERR_INVALID_ARG;
    }
    rumi_status st = ensure_workspace(sc, 256 + 3 * sizeof(unsigned long long) + 64 * sizeof(int));
    if (st != RUMI_OK) return st;
    if (uses_bvh8(trace_mode) && (st = ensure_bvh8(sc)) != RUMI_OK) return st;
    TraceLaunch T;
    T.s = sc->dev;
    T.rays = (const float4 *)rays_dev;
    T.t = t_dev;
    T.prim = prim_dev;
    T.n = n;
    T.anyhit = anyhit;
    T.counters = (unsigned long long *)sc->ws;
    cudaMemsetAsync(T.counters, 0, 3 * sizeof(unsigned long long) + 64 * sizeof(int), stream);
    if (n > 0) {
        const int m = trace_scheme(trace_mode);
        auto go = [&](auto mode_tag) {
            constexpr int M = decltype(mode_tag)::value;
            if (anyhit)
                launch_trace_batch<true, false, M>(T, sc->num_sms, stream);
            else
                launch_trace_batch<false, false, M>(T, sc->num_sms, stream);
        };
        switch (m) {
            case SCHEME_BATCH: go(std::integral_constant<int, SCHEME_BATCH>()); break;
            case SCHEME_REFILL: go(std::integral_constant<int, SCHEME_REFILL>()); break;
            case SCHEME_LEAVES: go(std::integral_constant<int, SCHEME_LEAVES>()); break;
            case SCHEME_WIDE: go(std::integral_constant<int, SCHEME_WIDE>()); break;
            default: go(std::integral_constant<int, SCHEME_EIGHT>()); break;
        }
    }
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return cuda_status(e, "trace_rays_scheme");
    return RUMI_OK;
}

#endif  // RUMI_HOST_BUILD

}  // namespace rumi
