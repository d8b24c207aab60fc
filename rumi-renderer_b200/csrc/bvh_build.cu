// On-device binned-SAH BVH build into 32-byte nodes.
//
// The reference builds an object-median BVH on the host (src/Acceleration/bvh.cpp:48-148:
// longest axis, shell sort, split at the middle index, leaves of <= 6).  Only the hits a
// BVH produces are observable, so this builder uses the surface area heuristic instead,
// entirely on the GPU and deterministically (same input -> same tree):
//
//  large phase (tasks with > SMALL_MAX primitives), one level per iteration:
//    bin           one block per chunk of CHUNK primitives: 3 axes x 32 centroid bins in shared
//                  memory, merged into the task's bins with global atomics (ordered-int floats)
//    split         one warp per task, lane = bin: prefix/suffix scans, SAH argmin; empties what
//                  this level's scatter and the next level's bin accumulate into
//    count/scan/scatter  stable partition into the other index array: per-chunk left counts,
//                  per-task scan, per-chunk block scan + scatter; child bounds by block reduction
//    level         one block: child nodes, the next level's tasks in order and their chunks,
//                  small tasks
//  small phase, one warp per task, the subtree built in shared memory (binned SAH, ballot-based
//    stable partition, explicit stack): first down to tasks of SMALL_MID primitives, then, a warp
//    for each of those, to the leaves.  (A warp that built a whole 256-primitive subtree was the
//    longest kernel of a build: 0.8 of 2.6 ms for 262k triangles, most SMs idle at its end.)
//
// No launch depends on a count that the host would have to read: grids are sized by what a level
// can hold and kernels stop at the device's counts.  The host looks once, after the expected
// number of levels and the small phase.
//
// Node index space: [0] root, [1] unused (pairs start 64-byte aligned), then one pair per split, at
// the position of its boundary in the primitive order (node 2 + 2 m for the split in front of
// primitive m, which no other split of the tree shares), then pairs for splits that leave a side
// empty.
#include "bvh_build.h"
#include <algorithm>
#include <cstdio>
#include <type_traits>

namespace rumi {

static constexpr int NBINS = 32;
static constexpr int CHUNK = 1024;
static constexpr int BIN_THREADS = 256;
static constexpr int PAIRS = 2;  // first node of the pair region
static constexpr int SMALL_MAX = 256;
static constexpr int SMALL_MID = 64;
// Bins per axis of the tasks of up to SMALL_MID primitives: with ten, the three axes' bins are the
// lanes of one warp and are scanned together (warp_sah_mid), a quarter of the work of three scans
// of 32: 262,154 triangles build in 1.43 ms, 1.68 with 32 bins there.  The trees, 32-byte node units +
// primitive tests per ray with ten / 32 bins: 18.2 + 10.7 both (displaced sphere), 79.2 / 79.0 + 23.8
// (200,000 triangles at random), 84.0 / 83.7 + 56.9 / 55.8 (50,000 that overlap), 345 / 344 + 366 / 359
// (needles), 64.5 / 64.4 + 11.8 (clusters), 10.0 + 10.3 both (a grid).
static constexpr int MID_BINS = 10;
// Leaf size cap and SAH traversal cost (relative to one primitive test).  Measured on the
// 1024x1024x64 BVH-bound frame (ms): cap 8 / C_TRAV 1: 239; cap 16 / 1: 239; 16 / 1.5: 250;
// 16, 24 or 32 / 2: 225.5; 16 / 3: 231; 8 / 2: 250 (larger leaves pay only when the cap
// lets the SAH form them).
#ifndef RUMI_LEAF_MAX
#define RUMI_LEAF_MAX 16
#endif
static constexpr int LEAF_MAX = RUMI_LEAF_MAX;
static constexpr int MEDIAN_DEPTH = 40;    // past this depth split at the index median
static constexpr int MAX_DEPTH = 63;       // deepest node (traversal stack holds 64)
#ifndef RUMI_SAH_CTRAV
#define RUMI_SAH_CTRAV 2.0f
#endif
static constexpr float C_TRAV = RUMI_SAH_CTRAV;
static constexpr float C_ISECT = 1.0f;

struct BuildTask {
    int first, count, node;
    int depth;  // a small task's depth carries the index array that holds it (IN_TMP)
};
static constexpr int IN_TMP = 1 << 20;

// Device counters of a build.
enum { K_LARGE = 0, K_LARGE1 = 1, K_SMALL = 2, K_CHUNKS = 3, K_ERR = 4, K_MID = 5, K_LEVELS = 6, K_SPARE = 7, K_NUM = 16 };
static_assert(K_NUM == BVH_COUNTERS, "bvh_wide reads these");
static_assert(BVH_DEFERRED <= SMALL_MAX, "no levels");

// Appends a task to one of the small phase's lists (n + 1 entries; a task per primitive at most,
// and empty sides of degenerate splits).
__device__ __forceinline__ void append_task(BuildTask *list, int *count, const BuildTask &t, int n, int *counters) {
    const int k = atomicAdd(count, 1);
    if (k <= n)
        list[k] = t;
    else
        atomicExch(counters + K_ERR, 5);
}

// Nodes of a split's two children: the pair of its boundary, or (a side is empty) a spare pair.
__device__ __forceinline__ int split_pair(int first, int nleft, int count, int n, int *counters) {
    if (nleft > 0 && nleft < count) return PAIRS + 2 * (first + nleft);
    return PAIRS + 2 * n + 2 * atomicAdd(counters + K_SPARE, 1);
}

struct Bounds12 {  // ordered ints: aabb lo/hi, centroid lo/hi
    int v[12];
};

// --------------------------------------------------------------------- helpers
__device__ __forceinline__ float area_of(float3 lo, float3 hi) {
    float3 e = hi - lo;
    if (e.x < 0.0f || e.y < 0.0f || e.z < 0.0f) return 0.0f;
    return 2.0f * (e.x * e.y + e.x * e.z + e.y * e.z);
}

__device__ __forceinline__ void pad_bounds(float3 &lo, float3 &hi) {
    // conservative padding so the float slab test never rejects a surface lying on a
    // box face
    const float ex = fmaxf(fabsf(lo.x), fabsf(hi.x)) * 9.5367431640625e-7f + 1e-30f;
    const float ey = fmaxf(fabsf(lo.y), fabsf(hi.y)) * 9.5367431640625e-7f + 1e-30f;
    const float ez = fmaxf(fabsf(lo.z), fabsf(hi.z)) * 9.5367431640625e-7f + 1e-30f;
    lo = mk3(lo.x - ex, lo.y - ey, lo.z - ez);
    hi = mk3(hi.x + ex, hi.y + ey, hi.z + ez);
}

__device__ __forceinline__ void write_node_bounds(BvhNode *nodes, int n, float3 lo, float3 hi) {
    pad_bounds(lo, hi);
    BvhNode &nd = nodes[n];
    nd.lo_x = lo.x; nd.lo_y = lo.y; nd.lo_z = lo.z;
    nd.hi_x = hi.x; nd.hi_y = hi.y; nd.hi_z = hi.z;
}

__device__ __forceinline__ int bin_of(float c, float cmin, float scale, int bins = NBINS) {
    int b = (int)((c - cmin) * scale);
    return b < 0 ? 0 : (b >= bins ? bins - 1 : b);
}

__device__ __forceinline__ float3 centroid(float4 lo, float4 hi) {
    return mk3((lo.x + hi.x) * 0.5f, (lo.y + hi.y) * 0.5f, (lo.z + hi.z) * 0.5f);
}

// ------------------------------------------------------------ primitive setup
// Bounds of every canonical primitive (from the original vertices, so they contain the
// triangle however its edges round) and its 48-byte intersection record.
__global__ void prim_prepare_kernel(const float *tri_v, int n_tris, const float4 *rects, int n_rects,
                                    const float4 *spheres, const int *prim_flags, int n_spheres,
                                    float4 *aabb_lo, float4 *aabb_hi, float4 *prims, int *idx, int *root_bounds) {
    const int N = n_tris + n_rects + n_spheres;
    float b[12];  // of this thread's primitives: box low / high, centroid low / high
    for (int j = 0; j < 12; ++j) b[j] = (j % 6) < 3 ? INFINITY : -INFINITY;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        float3 lo, hi;
        float4 A, B, C;
        if (i < n_tris) {
            const float *t = tri_v + 9 * (size_t)i;
            float3 v0 = mk3(t[0], t[1], t[2]), v1 = mk3(t[3], t[4], t[5]), v2 = mk3(t[6], t[7], t[8]);
            lo = mk3(fminf(v0.x, fminf(v1.x, v2.x)), fminf(v0.y, fminf(v1.y, v2.y)), fminf(v0.z, fminf(v1.z, v2.z)));
            hi = mk3(fmaxf(v0.x, fmaxf(v1.x, v2.x)), fmaxf(v0.y, fmaxf(v1.y, v2.y)), fmaxf(v0.z, fmaxf(v1.z, v2.z)));
            float3 e1 = rn_sub(v1, v0), e2 = rn_sub(v2, v0);
            A = make_float4(v0.x, v0.y, v0.z, __int_as_float(i));
            B = make_float4(e1.x, e1.y, e1.z, __int_as_float(PRIM_TRI));
            C = make_float4(e2.x, e2.y, e2.z, 0.0f);
        } else if (i < n_tris + n_rects) {
            const int r = i - n_tris;
            float4 p = rects[3 * r], l = rects[3 * r + 1], w = rects[3 * r + 2];
            float3 q = mk3(p.x + l.x + w.x, p.y + l.y + w.y, p.z + l.z + w.z);
            float3 pl = mk3(p.x + l.x, p.y + l.y, p.z + l.z), pw = mk3(p.x + w.x, p.y + w.y, p.z + w.z);
            lo = mk3(fminf(fminf(p.x, q.x), fminf(pl.x, pw.x)), fminf(fminf(p.y, q.y), fminf(pl.y, pw.y)),
                     fminf(fminf(p.z, q.z), fminf(pl.z, pw.z)));
            hi = mk3(fmaxf(fmaxf(p.x, q.x), fmaxf(pl.x, pw.x)), fmaxf(fmaxf(p.y, q.y), fmaxf(pl.y, pw.y)),
                     fmaxf(fmaxf(p.z, q.z), fmaxf(pl.z, pw.z)));
            A = make_float4(p.x, p.y, p.z, __int_as_float(i));
            B = make_float4(l.x, l.y, l.z, __int_as_float(PRIM_RECT | (prim_flags[r] ? PRIM_FLAG_EMISSIVE : 0)));
            C = make_float4(w.x, w.y, w.z, 0.0f);
        } else {
            const int s = i - n_tris - n_rects;
            float4 c = spheres[s];
            lo = mk3(c.x - c.w, c.y - c.w, c.z - c.w);
            hi = mk3(c.x + c.w, c.y + c.w, c.z + c.w);
            A = make_float4(c.x, c.y, c.z, __int_as_float(i));
            B = make_float4(c.w, 0.0f, 0.0f,
                            __int_as_float(PRIM_SPHERE | (prim_flags[n_rects + s] ? PRIM_FLAG_IBL : 0)));
            C = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        // a coordinate that is NaN in all vertices bounds nothing (NaN orders above all numbers in
        // the bins' integers, while the minima and maxima of floats drop it)
        lo = mk3(lo.x == lo.x ? lo.x : INFINITY, lo.y == lo.y ? lo.y : INFINITY, lo.z == lo.z ? lo.z : INFINITY);
        hi = mk3(hi.x == hi.x ? hi.x : -INFINITY, hi.y == hi.y ? hi.y : -INFINITY, hi.z == hi.z ? hi.z : -INFINITY);
        aabb_lo[i] = make_float4(lo.x, lo.y, lo.z, 0.0f);
        aabb_hi[i] = make_float4(hi.x, hi.y, hi.z, 0.0f);
        idx[i] = i;
        const float3 c = centroid(aabb_lo[i], aabb_hi[i]);
        b[0] = fminf(b[0], lo.x); b[1] = fminf(b[1], lo.y); b[2] = fminf(b[2], lo.z);
        b[3] = fmaxf(b[3], hi.x); b[4] = fmaxf(b[4], hi.y); b[5] = fmaxf(b[5], hi.z);
        b[6] = fminf(b[6], c.x); b[7] = fminf(b[7], c.y); b[8] = fminf(b[8], c.z);
        b[9] = fmaxf(b[9], c.x); b[10] = fmaxf(b[10], c.y); b[11] = fmaxf(b[11], c.z);
        prims[3 * (size_t)i + 0] = A;
        prims[3 * (size_t)i + 1] = B;
        prims[3 * (size_t)i + 2] = C;
    }
    __shared__ int s_b[12];
    if (threadIdx.x < 12) s_b[threadIdx.x] = (threadIdx.x % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    __syncthreads();
    for (int j = 0; j < 12; ++j) {
        const bool mx = (j % 6) >= 3;
        int v = f2o(b[j]);
        v = mx ? __reduce_max_sync(0xffffffffu, v) : __reduce_min_sync(0xffffffffu, v);
        if ((threadIdx.x & 31) == 0) {
            if (mx)
                atomicMax(s_b + j, v);
            else
                atomicMin(s_b + j, v);
        }
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        if ((threadIdx.x % 6) < 3)
            atomicMin(root_bounds + threadIdx.x, s_b[threadIdx.x]);
        else
            atomicMax(root_bounds + threadIdx.x, s_b[threadIdx.x]);
    }
}

__global__ void init_kernel(int *root_bounds, int *counters) {
    if (threadIdx.x < 12) root_bounds[threadIdx.x] = (threadIdx.x % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    if (threadIdx.x < K_NUM) counters[threadIdx.x] = 0;
}

struct ChunkInfo {
    int task;
    int start;   // absolute index into idx
    int len;
};

// One block: the chunks of `n_tasks` tasks (consecutive per task), and each task's first chunk.
__device__ void list_chunks(const BuildTask *tasks, int n_tasks, ChunkInfo *chunks, int *task_first_chunk, int *n_chunks) {
    __shared__ int s_scan[1024];
    __shared__ int s_base;
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    for (int t0 = 0; t0 < n_tasks; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        const int nc = t < n_tasks ? (tasks[t].count + CHUNK - 1) / CHUNK : 0;
        s_scan[threadIdx.x] = nc;
        __syncthreads();
        for (int o = 1; o < blockDim.x; o <<= 1) {
            int v = threadIdx.x >= o ? s_scan[threadIdx.x - o] : 0;
            __syncthreads();
            s_scan[threadIdx.x] += v;
            __syncthreads();
        }
        const int excl = s_scan[threadIdx.x] - nc + s_base;
        if (t < n_tasks) {
            const BuildTask tk = tasks[t];
            task_first_chunk[t] = excl;
            for (int c = 0; c < nc; ++c) {
                ChunkInfo ci;
                ci.task = t;
                ci.start = tk.first + c * CHUNK;
                ci.len = min(CHUNK, tk.count - c * CHUNK);
                chunks[excl + c] = ci;
            }
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) s_base = excl + nc;
        __syncthreads();
    }
    if (threadIdx.x == 0) *n_chunks = s_base;
}

__device__ __forceinline__ void empty_bins(int *bins, int from, int step) {
    for (int i = from; i < 3 * NBINS; i += step) {
        int *b = bins + 7 * i;
        b[0] = 0;
        b[1] = b[2] = b[3] = f2o(INFINITY);
        b[4] = b[5] = b[6] = f2o(-INFINITY);
    }
}

// Root node and root task (one block).
__global__ void root_kernel(const int *root_bounds, int n, BvhNode *nodes, BuildTask *large, int *cb, BuildTask *small,
                            BuildTask *mid, int *bins, ChunkInfo *chunks, int *task_first_chunk, int *counters) {
    if (threadIdx.x == 0) {
        if (n == 0) {
            BvhNode &r = nodes[0];
            r.lo_x = r.lo_y = r.lo_z = INFINITY;
            r.hi_x = r.hi_y = r.hi_z = -INFINITY;
            r.first = 0;
            r.count = 1;  // an empty leaf that is never entered
        } else {
            const int *b = root_bounds;
            write_node_bounds(nodes, 0, mk3(o2f(b[0]), o2f(b[1]), o2f(b[2])), mk3(o2f(b[3]), o2f(b[4]), o2f(b[5])));
            nodes[1] = nodes[0];
            nodes[1].count = -1;  // unused slot
            BuildTask t;
            t.first = 0; t.count = n; t.node = 0; t.depth = 0;
            if (n > SMALL_MAX) {
                large[0] = t;
                for (int j = 0; j < 6; ++j) cb[j] = b[6 + j];
                counters[K_LARGE] = 1;
            } else {
                small[0] = t;
                counters[K_SMALL] = 1;
                if (n <= SMALL_MID) {  // the first pass would only hand it on, and is not launched
                    mid[0] = t;
                    counters[K_MID] = 1;
                }
            }
        }
    }
    empty_bins(bins, threadIdx.x, blockDim.x);
    __syncthreads();
    if (n > SMALL_MAX) list_chunks(large, 1, chunks, task_first_chunk, counters + K_CHUNKS);
}

// ------------------------------------------------------------- large phase
// centroid bounds of each task, stored as ordered ints in cb[task][6]
__global__ void bin_kernel(const ChunkInfo *chunks, const int *n_chunks, const int *idx, const float4 *aabb_lo,
                           const float4 *aabb_hi, const int *cb, int *bins) {
    __shared__ int s_bins[3 * NBINS * 7];
    const int c = blockIdx.x;
    if (c >= *n_chunks) return;
    const ChunkInfo ci = chunks[c];
    empty_bins(s_bins, threadIdx.x, blockDim.x);
    __syncthreads();
    const int *tcb = cb + 6 * ci.task;
    const float cmin[3] = {o2f(tcb[0]), o2f(tcb[1]), o2f(tcb[2])};
    const float cmax[3] = {o2f(tcb[3]), o2f(tcb[4]), o2f(tcb[5])};
    float scale[3];
    for (int a = 0; a < 3; ++a) {
        const float ext = cmax[a] - cmin[a];
        scale[a] = ext > 0.0f ? (float)NBINS * (1.0f - 1e-6f) / ext : 0.0f;
    }
    for (int k = threadIdx.x; k < ci.len; k += blockDim.x) {
        const int p = idx[ci.start + k];
        const float4 lo = aabb_lo[p], hi = aabb_hi[p];
        const float3 cc = centroid(lo, hi);
        const float cv[3] = {cc.x, cc.y, cc.z};
        for (int a = 0; a < 3; ++a) {
            int *b = s_bins + 7 * (a * NBINS + bin_of(cv[a], cmin[a], scale[a]));
            atomicAdd(b, 1);
            atomicMin(b + 1, f2o(lo.x)); atomicMin(b + 2, f2o(lo.y)); atomicMin(b + 3, f2o(lo.z));
            atomicMax(b + 4, f2o(hi.x)); atomicMax(b + 5, f2o(hi.y)); atomicMax(b + 6, f2o(hi.z));
        }
    }
    __syncthreads();
    int *gb = bins + (size_t)ci.task * 3 * NBINS * 7;
    for (int i = threadIdx.x; i < 3 * NBINS; i += blockDim.x) {
        const int *b = s_bins + 7 * i;
        if (b[0] == 0) continue;
        int *g = gb + 7 * i;
        atomicAdd(g, b[0]);
        atomicMin(g + 1, b[1]); atomicMin(g + 2, b[2]); atomicMin(g + 3, b[3]);
        atomicMax(g + 4, b[4]); atomicMax(g + 5, b[5]); atomicMax(g + 6, b[6]);
    }
}

struct SplitDecision {
    int axis;   // -1: index-median split
    int bin;    // primitives with bin <= this go left
    int nleft;
};

// Warp-level SAH sweep over 32 bins of three axes: lane j owns bin j.  Returns the best
// (cost, axis, bin, nleft) in every lane; cost = INF when no bin split separates anything.
__device__ void warp_sah(const int *bins /* [3][NBINS][7] */, float &best_cost, int &best_axis, int &best_bin,
                         int &best_nleft) {
    const int lane = threadIdx.x & 31;
    best_cost = INFINITY;
    best_axis = -1;
    best_bin = 0;
    best_nleft = 0;
    for (int a = 0; a < 3; ++a) {
        const int *b = bins + 7 * (a * NBINS + lane);
        int cnt = b[0];
        float lx = o2f(b[1]), ly = o2f(b[2]), lz = o2f(b[3]);
        float hx = o2f(b[4]), hy = o2f(b[5]), hz = o2f(b[6]);
        // inclusive prefix (left side ending at bin lane)
        int pc = cnt;
        float plx = lx, ply = ly, plz = lz, phx = hx, phy = hy, phz = hz;
        for (int o = 1; o < 32; o <<= 1) {
            int c2 = __shfl_up_sync(0xffffffffu, pc, o);
            float a0 = __shfl_up_sync(0xffffffffu, plx, o), a1 = __shfl_up_sync(0xffffffffu, ply, o);
            float a2 = __shfl_up_sync(0xffffffffu, plz, o), a3 = __shfl_up_sync(0xffffffffu, phx, o);
            float a4 = __shfl_up_sync(0xffffffffu, phy, o), a5 = __shfl_up_sync(0xffffffffu, phz, o);
            if (lane >= o) {
                pc += c2;
                plx = fminf(plx, a0); ply = fminf(ply, a1); plz = fminf(plz, a2);
                phx = fmaxf(phx, a3); phy = fmaxf(phy, a4); phz = fmaxf(phz, a5);
            }
        }
        // inclusive suffix (right side starting at bin lane)
        int sc = cnt;
        float slx = lx, sly = ly, slz = lz, shx = hx, shy = hy, shz = hz;
        for (int o = 1; o < 32; o <<= 1) {
            int c2 = __shfl_down_sync(0xffffffffu, sc, o);
            float a0 = __shfl_down_sync(0xffffffffu, slx, o), a1 = __shfl_down_sync(0xffffffffu, sly, o);
            float a2 = __shfl_down_sync(0xffffffffu, slz, o), a3 = __shfl_down_sync(0xffffffffu, shx, o);
            float a4 = __shfl_down_sync(0xffffffffu, shy, o), a5 = __shfl_down_sync(0xffffffffu, shz, o);
            if (lane + o < 32) {
                sc += c2;
                slx = fminf(slx, a0); sly = fminf(sly, a1); slz = fminf(slz, a2);
                shx = fmaxf(shx, a3); shy = fmaxf(shy, a4); shz = fmaxf(shz, a5);
            }
        }
        // right side of a split after bin lane = suffix of lane+1
        int rc = __shfl_down_sync(0xffffffffu, sc, 1);
        float r0 = __shfl_down_sync(0xffffffffu, slx, 1), r1 = __shfl_down_sync(0xffffffffu, sly, 1);
        float r2 = __shfl_down_sync(0xffffffffu, slz, 1), r3 = __shfl_down_sync(0xffffffffu, shx, 1);
        float r4 = __shfl_down_sync(0xffffffffu, shy, 1), r5 = __shfl_down_sync(0xffffffffu, shz, 1);
        float cost = INFINITY;
        if (lane < 31 && pc > 0 && rc > 0) {
            cost = area_of(mk3(plx, ply, plz), mk3(phx, phy, phz)) * (float)pc +
                   area_of(mk3(r0, r1, r2), mk3(r3, r4, r5)) * (float)rc;
        }
        // warp argmin (ties -> lowest lane)
        float bc = cost;
        int bl = lane;
        for (int o = 16; o > 0; o >>= 1) {
            float oc = __shfl_xor_sync(0xffffffffu, bc, o);
            int ol = __shfl_xor_sync(0xffffffffu, bl, o);
            if (oc < bc || (oc == bc && ol < bl)) {
                bc = oc;
                bl = ol;
            }
        }
        const int nl = __shfl_sync(0xffffffffu, pc, bl);
        if (bc < best_cost) {
            best_cost = bc;
            best_axis = a;
            best_bin = bl;
            best_nleft = nl;
        }
    }
}

// The same over MID_BINS bins of three axes, lane = 10 axis + bin.  Every lane also receives the
// bounds of the two sides of the best split.
__device__ void warp_sah_mid(const int *bins /* [3][MID_BINS][7] */, float &best_cost, int &best_axis, int &best_bin,
                             int &best_nleft, float3 lo[2], float3 hi[2]) {
    const int lane = threadIdx.x & 31, axis = lane / MID_BINS, bin = lane - axis * MID_BINS;
    const bool on = axis < 3;
    const int *b = bins + 7 * (on ? lane : 0);
    int pc = on ? b[0] : 0;
    float p[6], q[6];  // this bin and those before it / after it: low, high
    for (int j = 0; j < 6; ++j) p[j] = q[j] = on ? o2f(b[1 + j]) : (j < 3 ? INFINITY : -INFINITY);
    int sc = pc;
    for (int o = 1; o < MID_BINS; o <<= 1) {
        const int c1 = __shfl_up_sync(0xffffffffu, pc, o), c2 = __shfl_down_sync(0xffffffffu, sc, o);
        float u[6], d[6];
        for (int j = 0; j < 6; ++j) {
            u[j] = __shfl_up_sync(0xffffffffu, p[j], o);
            d[j] = __shfl_down_sync(0xffffffffu, q[j], o);
        }
        if (bin >= o) {
            pc += c1;
            for (int j = 0; j < 6; ++j) p[j] = j < 3 ? fminf(p[j], u[j]) : fmaxf(p[j], u[j]);
        }
        if (bin + o < MID_BINS && on) {
            sc += c2;
            for (int j = 0; j < 6; ++j) q[j] = j < 3 ? fminf(q[j], d[j]) : fmaxf(q[j], d[j]);
        }
    }
    // the right side of a split after this bin
    const int rc = __shfl_down_sync(0xffffffffu, sc, 1);
    for (int j = 0; j < 6; ++j) q[j] = __shfl_down_sync(0xffffffffu, q[j], 1);
    float cost = INFINITY;
    if (on && bin < MID_BINS - 1 && pc > 0 && rc > 0)
        cost = area_of(mk3(p[0], p[1], p[2]), mk3(p[3], p[4], p[5])) * (float)pc +
               area_of(mk3(q[0], q[1], q[2]), mk3(q[3], q[4], q[5])) * (float)rc;
    // costs are not negative, so their bits order like them; ties go to the lowest lane
    const int least = __reduce_min_sync(0xffffffffu, __float_as_int(cost));
    const unsigned at = __ballot_sync(0xffffffffu, __float_as_int(cost) == least);
    const int best = __ffs(at) - 1;
    best_cost = __int_as_float(least);
    best_axis = best_cost < INFINITY ? best / MID_BINS : -1;
    best_bin = best - (best / MID_BINS) * MID_BINS;
    best_nleft = __shfl_sync(0xffffffffu, pc, best);
    lo[0] = mk3(__shfl_sync(0xffffffffu, p[0], best), __shfl_sync(0xffffffffu, p[1], best), __shfl_sync(0xffffffffu, p[2], best));
    hi[0] = mk3(__shfl_sync(0xffffffffu, p[3], best), __shfl_sync(0xffffffffu, p[4], best), __shfl_sync(0xffffffffu, p[5], best));
    lo[1] = mk3(__shfl_sync(0xffffffffu, q[0], best), __shfl_sync(0xffffffffu, q[1], best), __shfl_sync(0xffffffffu, q[2], best));
    hi[1] = mk3(__shfl_sync(0xffffffffu, q[3], best), __shfl_sync(0xffffffffu, q[4], best), __shfl_sync(0xffffffffu, q[5], best));
}

// next_bins: the other level's bins, emptied here for the children of every task.
__global__ void split_kernel(const BuildTask *tasks, const int *n_tasks, const int *bins, int *next_bins, int max_tasks,
                             int *child_bounds, SplitDecision *dec) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= *n_tasks) return;
    const int lane = threadIdx.x & 31;
    if (lane < 24) child_bounds[24 * t + lane] = (lane % 6) < 3 ? f2o(INFINITY) : f2o(-INFINITY);
    for (int k = 2 * t; k < 2 * t + 2 && k < max_tasks; ++k) empty_bins(next_bins + (size_t)k * 3 * NBINS * 7, lane, 32);
    const BuildTask tk = tasks[t];
    float cost;
    int axis, bin, nl;
    warp_sah(bins + (size_t)t * 3 * NBINS * 7, cost, axis, bin, nl);
    if ((threadIdx.x & 31) == 0) {
        SplitDecision d;
        if (axis < 0 || tk.depth >= MEDIAN_DEPTH) {
            d.axis = -1;
            d.bin = 0;
            d.nleft = tk.count / 2;
        } else {
            d.axis = axis;
            d.bin = bin;
            d.nleft = nl;
        }
        dec[t] = d;
    }
}

__device__ __forceinline__ bool goes_left(const SplitDecision &d, int pos_in_task, float3 c, const int *tcb) {
    if (d.axis < 0) return pos_in_task < d.nleft;
    const float cv = d.axis == 0 ? c.x : (d.axis == 1 ? c.y : c.z);
    const float cmin = o2f(tcb[d.axis]), cmax = o2f(tcb[3 + d.axis]);
    const float ext = cmax - cmin;
    const float scale = ext > 0.0f ? (float)NBINS * (1.0f - 1e-6f) / ext : 0.0f;
    return bin_of(cv, cmin, scale) <= d.bin;
}

static constexpr int PER_THREAD = CHUNK / BIN_THREADS;

__global__ void count_kernel(const ChunkInfo *chunks, const int *n_chunks, const BuildTask *tasks,
                             const SplitDecision *dec, const int *idx, const float4 *aabb_lo, const float4 *aabb_hi,
                             const int *cb, int *chunk_left) {
    __shared__ int s_red[BIN_THREADS / 32];
    const int c = blockIdx.x;
    if (c >= *n_chunks) return;
    const ChunkInfo ci = chunks[c];
    const BuildTask tk = tasks[ci.task];
    const SplitDecision d = dec[ci.task];
    const int *tcb = cb + 6 * ci.task;
    int cnt = 0;
    for (int k = threadIdx.x; k < ci.len; k += blockDim.x) {
        const int pos = ci.start + k;
        const int p = idx[pos];
        const float3 cc = centroid(aabb_lo[p], aabb_hi[p]);
        cnt += goes_left(d, pos - tk.first, cc, tcb) ? 1 : 0;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int i = 0; i < BIN_THREADS / 32; ++i) s += s_red[i];
        chunk_left[c] = s;
    }
}

// One warp per task: exclusive scan of its chunks' left counts (chunks of a task are
// consecutive in the chunk list).
__global__ void chunk_scan_kernel(const ChunkInfo *chunks, const int *n_chunks, const int *n_tasks,
                                  const int *chunk_left, int *chunk_loff, const int *task_first_chunk,
                                  SplitDecision *dec) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= *n_tasks) return;
    const int c0 = task_first_chunk[t];
    const int nch = *n_chunks;
    int running = 0;
    for (int base = c0;; base += 32) {
        const int c = base + lane;
        const bool valid = c < nch && chunks[c].task == t;
        int v = valid ? chunk_left[c] : 0;
        int incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            int x = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += x;
        }
        if (valid) chunk_loff[c] = running + incl - v;
        running += __shfl_sync(0xffffffffu, incl, 31);
        const unsigned any_invalid = __ballot_sync(0xffffffffu, !valid);
        if (any_invalid) break;
    }
    if (lane == 0) dec[t].nleft = running;  // exact left count of the partition
}

__global__ void scatter_kernel(const ChunkInfo *chunks, const int *n_chunks, const BuildTask *tasks,
                               const SplitDecision *dec, const int *idx, int *idx_tmp, const float4 *aabb_lo,
                               const float4 *aabb_hi, const int *cb, const int *chunk_loff, int *child_bounds) {
    __shared__ int s_scan[BIN_THREADS];
    __shared__ int s_b[2][12][BIN_THREADS / 32];
    const int c = blockIdx.x;
    if (c >= *n_chunks) return;
    const ChunkInfo ci = chunks[c];
    const BuildTask tk = tasks[ci.task];
    const SplitDecision d = dec[ci.task];
    const int *tcb = cb + 6 * ci.task;
    const int k0 = threadIdx.x * PER_THREAD;
    int pidx[PER_THREAD];
    bool left[PER_THREAD];
    int nl = 0;
    float bl[2][12];
    for (int s = 0; s < 2; ++s)
        for (int j = 0; j < 12; ++j) bl[s][j] = (j % 6) < 3 ? INFINITY : -INFINITY;
    for (int k = 0; k < PER_THREAD; ++k) {
        const int kk = k0 + k;
        left[k] = false;
        pidx[k] = -1;
        if (kk < ci.len) {
            const int pos = ci.start + kk;
            const int p = idx[pos];
            const float4 lo = aabb_lo[p], hi = aabb_hi[p];
            const float3 cc = centroid(lo, hi);
            const bool L = goes_left(d, pos - tk.first, cc, tcb);
            pidx[k] = p;
            left[k] = L;
            nl += L;
            float *b = bl[L ? 0 : 1];
            b[0] = fminf(b[0], lo.x); b[1] = fminf(b[1], lo.y); b[2] = fminf(b[2], lo.z);
            b[3] = fmaxf(b[3], hi.x); b[4] = fmaxf(b[4], hi.y); b[5] = fmaxf(b[5], hi.z);
            b[6] = fminf(b[6], cc.x); b[7] = fminf(b[7], cc.y); b[8] = fminf(b[8], cc.z);
            b[9] = fmaxf(b[9], cc.x); b[10] = fmaxf(b[10], cc.y); b[11] = fmaxf(b[11], cc.z);
        }
    }
    // block exclusive scan of nl
    s_scan[threadIdx.x] = nl;
    __syncthreads();
    for (int o = 1; o < BIN_THREADS; o <<= 1) {
        int v = threadIdx.x >= o ? s_scan[threadIdx.x - o] : 0;
        __syncthreads();
        s_scan[threadIdx.x] += v;
        __syncthreads();
    }
    const int lrank = s_scan[threadIdx.x] - nl;
    const int chunk_off = ci.start - tk.first;          // primitives of this task before the chunk
    const int loff = chunk_loff[c];
    const int roff = chunk_off - loff;                  // right primitives before the chunk
    const int my_off = k0;                              // primitives of this chunk before my first
    int li = lrank, ri = my_off - lrank;
    for (int k = 0; k < PER_THREAD; ++k) {
        if (pidx[k] < 0) continue;
        int dst;
        if (left[k])
            dst = tk.first + loff + li++;
        else
            dst = tk.first + d.nleft + roff + ri++;
        if (dst >= tk.first && dst < tk.first + tk.count) idx_tmp[dst] = pidx[k];
    }
    // child bounds: warp reduce then block reduce then global atomics
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int s = 0; s < 2; ++s)
        for (int j = 0; j < 12; ++j) {
            float v = bl[s][j];
            const bool mx = (j % 6) >= 3;
            for (int o = 16; o > 0; o >>= 1) {
                float x = __shfl_xor_sync(0xffffffffu, v, o);
                v = mx ? fmaxf(v, x) : fminf(v, x);
            }
            if (lane == 0) s_b[s][j][w] = __float_as_int(v);
        }
    __syncthreads();
    if (threadIdx.x < 24) {
        const int s = threadIdx.x / 12, j = threadIdx.x % 12;
        const bool mx = (j % 6) >= 3;
        float v = __int_as_float(s_b[s][j][0]);
        for (int i = 1; i < BIN_THREADS / 32; ++i) {
            float x = __int_as_float(s_b[s][j][i]);
            v = mx ? fmaxf(v, x) : fminf(v, x);
        }
        int *g = child_bounds + 12 * (2 * ci.task + s) + j;
        if (mx)
            atomicMax(g, f2o(v));
        else
            atomicMin(g, f2o(v));
    }
}

// One block: the children of every large task (node pair, bounds), the next level's tasks (large
// children in order, so that the task order and with it the build is deterministic) with their
// centroid bounds and chunks, and small tasks, appended in any order (each builds only the nodes
// and index range of its own primitives).  in_tmp: which index array this level's scatter filled.
__global__ void level_kernel(const BuildTask *tasks, int *n_tasks_p, const SplitDecision *dec, const int *child_bounds,
                             int n, int max_nodes, BvhNode *nodes, BuildTask *next, int *next_cb, int *n_next, BuildTask *small,
                             int in_tmp, ChunkInfo *chunks, int *task_first_chunk, int *counters) {
    __shared__ int s_warp[32];
    __shared__ int s_base;
    const int n_tasks = *n_tasks_p;
    if (n_tasks == 0) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_base = 0;
        ++counters[K_LEVELS];
    }
    __syncthreads();
    for (int i0 = 0; i0 < 2 * n_tasks; i0 += blockDim.x) {  // thread = child i = 2 task + side
        const int i = i0 + threadIdx.x;
        const bool here = i < 2 * n_tasks;
        BuildTask ch;
        const int *b = child_bounds + 12 * (size_t)i;
        bool large = false;
        int pair = 0;
        if (here && (i & 1) == 0) {
            const BuildTask tk = tasks[i >> 1];
            pair = split_pair(tk.first, dec[i >> 1].nleft, tk.count, n, counters);
            if (pair + 1 >= max_nodes) {
                atomicExch(counters + K_ERR, 4);
                pair = 0;
            } else {
                nodes[tk.node].first = pair;
                nodes[tk.node].count = 0;
            }
        }
        pair = __shfl_sync(0xffffffffu, pair, lane & ~1);
        if (here && pair > 0) {
            const BuildTask tk = tasks[i >> 1];
            const int nleft = dec[i >> 1].nleft, side = i & 1;
            ch.first = side == 0 ? tk.first : tk.first + nleft;
            ch.count = side == 0 ? nleft : tk.count - nleft;
            ch.node = pair + side;
            ch.depth = tk.depth + 1;
            write_node_bounds(nodes, ch.node, mk3(o2f(b[0]), o2f(b[1]), o2f(b[2])), mk3(o2f(b[3]), o2f(b[4]), o2f(b[5])));
            nodes[ch.node].first = 0;
            nodes[ch.node].count = 0;
            large = ch.count > SMALL_MAX;
            if (!large) {
                ch.depth |= in_tmp ? IN_TMP : 0;
                append_task(small, counters + K_SMALL, ch, n, counters);
            }
        }
        // ordered compaction of the large children
        const unsigned m = __ballot_sync(0xffffffffu, large);
        if (lane == 0) s_warp[w] = __popc(m);
        __syncthreads();
        int before = 0, total = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
            if (k < w) before += s_warp[k];
            total += s_warp[k];
        }
        if (large) {
            const int dst = s_base + before + __popc(m & ((1u << lane) - 1u));
            next[dst] = ch;
            for (int j = 0; j < 6; ++j) next_cb[6 * dst + j] = b[6 + j];
        }
        __syncthreads();
        if (threadIdx.x == 0) s_base += total;
        __syncthreads();
    }
    const int m = s_base;
    if (threadIdx.x == 0) {
        *n_next = m;
        *n_tasks_p = 0;  // counts the level after next
    }
    list_chunks(next, m, chunks, task_first_chunk, counters + K_CHUNKS);
}

// ------------------------------------------------------------- small phase
static constexpr int SMALL_WARPS = 4;
static constexpr int SMALL_STACK = 24;

// Minimum of lo / maximum of hi over the warp, in every lane.
__device__ __forceinline__ void warp_bounds(float3 &lo, float3 &hi) {
    lo = mk3(o2f(__reduce_min_sync(0xffffffffu, f2o(lo.x))), o2f(__reduce_min_sync(0xffffffffu, f2o(lo.y))),
             o2f(__reduce_min_sync(0xffffffffu, f2o(lo.z))));
    hi = mk3(o2f(__reduce_max_sync(0xffffffffu, f2o(hi.x))), o2f(__reduce_max_sync(0xffffffffu, f2o(hi.y))),
             o2f(__reduce_max_sync(0xffffffffu, f2o(hi.z))));
}

// Subtrees of the list's tasks from `begin` on.  MAX: primitives of a task.  mid != nullptr: children of
// up to SMALL_MID primitives become tasks of the second pass instead of being built here.
template <int MAX>
__global__ void __launch_bounds__(32 * SMALL_WARPS) small_build_kernel(const BuildTask *small, const int *n_small, int begin, int n,
                                                                        int *idx, const int *idx_tmp, const float4 *aabb_lo,
                                                                        const float4 *aabb_hi, BvhNode *nodes, int max_nodes,
                                                                        BuildTask *mid, int *counters) {
    __shared__ int s_idx[SMALL_WARPS][MAX];
    __shared__ int s_tmp[SMALL_WARPS][MAX];
    constexpr bool MID = MAX <= SMALL_MID;
    constexpr int BINS = MID ? MID_BINS : NBINS;
    __shared__ int s_bins[SMALL_WARPS][3 * BINS * 7];
    int *error_flag = counters + K_ERR;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *sidx = s_idx[w];
    int *stmp = s_tmp[w];
    int *sb = s_bins[w];
    const int n_tasks = min(*n_small, n + 1);
    for (int t = begin + blockIdx.x * SMALL_WARPS + w; t < n_tasks; t += gridDim.x * SMALL_WARPS) {
        __syncwarp();
        BuildTask root = small[t];
        const int *src = (root.depth & IN_TMP) ? idx_tmp : idx;
        root.depth &= ~IN_TMP;
        for (int k = lane; k < root.count; k += 32) sidx[k] = src[root.first + k];
        __syncwarp();
        if (mid && root.count <= SMALL_MID) {
            for (int k = lane; k < root.count; k += 32) idx[root.first + k] = sidx[k];
            if (lane == 0) append_task(mid, counters + K_MID, root, n, counters);
            continue;
        }
        // stack entries: off, count, node, depth
        int st_off[SMALL_STACK], st_cnt[SMALL_STACK], st_node[SMALL_STACK], st_dep[SMALL_STACK];
        int sp = 0;
        int off = 0, cnt = root.count, node = root.node, dep = root.depth;
        for (;;) {
            // centroid bounds of this sub-range
            float3 cmn = mk3(INFINITY, INFINITY, INFINITY), cmx = mk3(-INFINITY, -INFINITY, -INFINITY);
            for (int k = lane; k < cnt; k += 32) {
                const int p = sidx[off + k];
                const float3 c = centroid(aabb_lo[p], aabb_hi[p]);
                cmn = mk3(fminf(cmn.x, c.x), fminf(cmn.y, c.y), fminf(cmn.z, c.z));
                cmx = mk3(fmaxf(cmx.x, c.x), fmaxf(cmx.y, c.y), fmaxf(cmx.z, c.z));
            }
            warp_bounds(cmn, cmx);
            bool make_leaf = cnt <= 1 || dep >= MAX_DEPTH;
            float best_cost = INFINITY;
            int axis = -1, bin = 0, nleft = cnt / 2;
            const float cminv[3] = {cmn.x, cmn.y, cmn.z}, cmaxv[3] = {cmx.x, cmx.y, cmx.z};
            float scale[3];
            float3 side_lo[2], side_hi[2];  // of the best split's sides (MID)
            for (int a = 0; a < 3; ++a) {
                const float ext = cmaxv[a] - cminv[a];
                scale[a] = ext > 0.0f ? (float)BINS * (1.0f - 1e-6f) / ext : 0.0f;
            }
            if (!make_leaf) {
                for (int i = lane; i < 3 * BINS; i += 32) {
                    sb[7 * i + 0] = 0;
                    sb[7 * i + 1] = sb[7 * i + 2] = sb[7 * i + 3] = f2o(INFINITY);
                    sb[7 * i + 4] = sb[7 * i + 5] = sb[7 * i + 6] = f2o(-INFINITY);
                }
                __syncwarp();
                for (int k = lane; k < cnt; k += 32) {
                    const int p = sidx[off + k];
                    const float4 lo = aabb_lo[p], hi = aabb_hi[p];
                    const float3 c = centroid(lo, hi);
                    const float cv[3] = {c.x, c.y, c.z};
                    for (int a = 0; a < 3; ++a) {
                        int *b = sb + 7 * (a * BINS + bin_of(cv[a], cminv[a], scale[a], BINS));
                        atomicAdd(b, 1);
                        atomicMin(b + 1, f2o(lo.x)); atomicMin(b + 2, f2o(lo.y)); atomicMin(b + 3, f2o(lo.z));
                        atomicMax(b + 4, f2o(hi.x)); atomicMax(b + 5, f2o(hi.y)); atomicMax(b + 6, f2o(hi.z));
                    }
                }
                __syncwarp();
                int bx, bb, bn;
                if constexpr (MID)
                    warp_sah_mid(sb, best_cost, bx, bb, bn, side_lo, side_hi);
                else
                    warp_sah(sb, best_cost, bx, bb, bn);
                const BvhNode &nd = nodes[node];
                const float parent_area = area_of(mk3(nd.lo_x, nd.lo_y, nd.lo_z), mk3(nd.hi_x, nd.hi_y, nd.hi_z));
                if (bx >= 0 && dep < MEDIAN_DEPTH) {
                    const float split_cost = C_TRAV + C_ISECT * best_cost / fmaxf(parent_area, 1e-30f);
                    const float leaf_cost = C_ISECT * (float)cnt;
                    if (cnt <= LEAF_MAX && leaf_cost <= split_cost) make_leaf = true;
                    axis = bx;
                    bin = bb;
                    nleft = bn;
                } else if (cnt <= 2 || (bx < 0 && cnt <= LEAF_MAX)) {
                    make_leaf = true;
                }
            }
            if (make_leaf) {
                if (lane == 0) {
                    nodes[node].first = root.first + off;
                    nodes[node].count = cnt;
                }
            } else {
                // stable partition of sidx[off, off+cnt) by the decision
                int lbase = 0, rbase = 0;
                for (int g = 0; g < cnt; g += 32) {
                    const int k = g + lane;
                    bool L = false;
                    int p = -1;
                    if (k < cnt) {
                        p = sidx[off + k];
                        if (axis < 0) {
                            L = k < nleft;
                        } else {
                            const float3 c = centroid(aabb_lo[p], aabb_hi[p]);
                            const float cv = axis == 0 ? c.x : (axis == 1 ? c.y : c.z);
                            L = bin_of(cv, cminv[axis], scale[axis], BINS) <= bin;
                        }
                    }
                    const unsigned bl = __ballot_sync(0xffffffffu, k < cnt && L);
                    const unsigned br = __ballot_sync(0xffffffffu, k < cnt && !L);
                    const unsigned lt = (1u << lane) - 1u;
                    if (k < cnt) {
                        const int dst = L ? off + lbase + __popc(bl & lt) : off + nleft + rbase + __popc(br & lt);
                        if (dst >= off && dst < off + cnt)
                            stmp[dst] = p;
                        else
                            atomicExch(error_flag, 2);
                    }
                    lbase += __popc(bl);
                    rbase += __popc(br);
                }
                __syncwarp();
                for (int k = lane; k < cnt; k += 32) sidx[off + k] = stmp[off + k];
                __syncwarp();
                // child bounds
                int pair = 0;
                if (lane == 0) pair = split_pair(root.first + off, nleft, cnt, n, counters);
                pair = __shfl_sync(0xffffffffu, pair, 0);
                if (pair + 1 >= max_nodes) {  // cannot happen: a pair per boundary
                    if (lane == 0) {
                        atomicExch(error_flag, 3);
                        nodes[node].first = root.first + off;
                        nodes[node].count = cnt;
                    }
                    __syncwarp();
                    if (sp == 0) break;
                    --sp;
                    off = st_off[sp]; cnt = st_cnt[sp]; node = st_node[sp]; dep = st_dep[sp];
                    continue;
                }
                for (int s = 0; s < 2; ++s) {
                    const int o2 = s == 0 ? off : off + nleft;
                    const int c2 = s == 0 ? nleft : cnt - nleft;
                    float3 lo = mk3(INFINITY, INFINITY, INFINITY), hi = mk3(-INFINITY, -INFINITY, -INFINITY);
                    if (MID && axis >= 0) {
                        lo = side_lo[s];
                        hi = side_hi[s];
                    } else {
                        for (int k = lane; k < c2; k += 32) {
                            const int p = sidx[o2 + k];
                            const float4 a = aabb_lo[p], b = aabb_hi[p];
                            lo = mk3(fminf(lo.x, a.x), fminf(lo.y, a.y), fminf(lo.z, a.z));
                            hi = mk3(fmaxf(hi.x, b.x), fmaxf(hi.y, b.y), fmaxf(hi.z, b.z));
                        }
                        warp_bounds(lo, hi);
                    }
                    if (lane == 0) {
                        write_node_bounds(nodes, pair + s, lo, hi);
                        nodes[pair + s].first = 0;
                        nodes[pair + s].count = 0;
                    }
                }
                if (lane == 0) {
                    nodes[node].first = pair;
                    nodes[node].count = 0;
                }
                // continue with the smaller child, push the larger one
                const int lc = nleft, rc = cnt - nleft;
                const bool left_small = lc <= rc;
                const int so = left_small ? off : off + nleft, sc = left_small ? lc : rc, sn = left_small ? pair : pair + 1;
                const int bo = left_small ? off + nleft : off, bc = left_small ? rc : lc, bn = left_small ? pair + 1 : pair;
                if (mid && sc <= SMALL_MID) {  // (the smaller child first, so a deferred larger one implies it)
                    if (lane == 0) append_task(mid, counters + K_MID, BuildTask{root.first + so, sc, sn, dep + 1}, n, counters);
                    if (bc <= SMALL_MID) {
                        if (lane == 0) append_task(mid, counters + K_MID, BuildTask{root.first + bo, bc, bn, dep + 1}, n, counters);
                        __syncwarp();
                        if (sp == 0) break;
                        --sp;
                        off = st_off[sp]; cnt = st_cnt[sp]; node = st_node[sp]; dep = st_dep[sp];
                        continue;
                    }
                    off = bo; cnt = bc; node = bn; dep = dep + 1;
                    __syncwarp();
                    continue;
                }
                if (sp < SMALL_STACK) {
                    st_off[sp] = bo; st_cnt[sp] = bc; st_node[sp] = bn; st_dep[sp] = dep + 1;
                    ++sp;
                } else {
                    // cannot happen (stack depth <= log2(SMALL_MAX)); record and make a leaf
                    if (lane == 0) {
                        atomicExch(error_flag, 1);
                        nodes[bn].first = root.first + bo;
                        nodes[bn].count = bc;
                    }
                }
                off = so; cnt = sc; node = sn; dep = dep + 1;
                __syncwarp();
                continue;
            }
            __syncwarp();
            if (sp == 0) break;
            --sp;
            off = st_off[sp]; cnt = st_cnt[sp]; node = st_node[sp]; dep = st_dep[sp];
        }
        __syncwarp();
        for (int k = lane; k < root.count; k += 32) idx[root.first + k] = sidx[k];
    }
}

__global__ void gather_leaf_prims_kernel(const int *idx, int n, const float4 *prims_canon, float4 *leaf_prims) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = idx[i];
        leaf_prims[3 * (size_t)i + 0] = prims_canon[3 * (size_t)p + 0];
        leaf_prims[3 * (size_t)i + 1] = prims_canon[3 * (size_t)p + 1];
        leaf_prims[3 * (size_t)i + 2] = prims_canon[3 * (size_t)p + 2];
    }
}

// ---------------------------------------------------------------- host driver
static inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

int bvh_node_capacity(int n_prims) {
    const long long n = n_prims;
    // root + pad, a pair per boundary, and spare pairs for splits that leave a side empty: at most
    // one per task and level
    long long cap = PAIRS + 2 * n + 2 * (n / SMALL_MAX + 1) * 64 + 64;
    return (int)cap;
}

// The build's arrays in its scratch memory.
struct BuildArrays {
    float4 *aabb_lo, *aabb_hi, *prims_canon;
    int *idx[2];
    BuildTask *tasks[2], *small, *mid;
    int *cbs[2], *bins[2], *child_bounds;
    ChunkInfo *chunks;
    int *chunk_left, *chunk_loff, *task_first_chunk;
    SplitDecision *dec;
    int *root_bounds, *counters;
};

static size_t carve_build(BuildArrays &B, char *base, int n_prims) {
    const size_t n = (size_t)(n_prims > 0 ? n_prims : 1);
    const size_t max_tasks = n / SMALL_MAX + 2;
    const size_t max_chunks = n / CHUNK + max_tasks + 2;
    char *p = base;
    auto take = [&](auto *&dst, size_t count) {
        dst = reinterpret_cast<std::remove_reference_t<decltype(dst)>>(p);
        p += (count * sizeof(*dst) + 255) & ~(size_t)255;
    };
    take(B.aabb_lo, n);
    take(B.aabb_hi, n);
    take(B.prims_canon, 3 * n);
    take(B.idx[0], n);
    take(B.idx[1], n);
    for (int k = 0; k < 2; ++k) {
        take(B.tasks[k], max_tasks);
        take(B.cbs[k], max_tasks * 6);
        take(B.bins[k], max_tasks * 3 * NBINS * 7);
    }
    take(B.small, n + 1);
    take(B.mid, n + 1);
    take(B.child_bounds, 2 * max_tasks * 12);
    take(B.chunks, max_chunks);
    take(B.chunk_left, max_chunks);
    take(B.chunk_loff, max_chunks);
    take(B.task_first_chunk, max_tasks);
    take(B.dec, max_tasks);
    take(B.root_bounds, 12);
    take(B.counters, K_NUM);
    return (size_t)(p - base);
}

size_t bvh_scratch_bytes(int n_prims) {
    BuildArrays B;
    return carve_build(B, nullptr, n_prims);
}

// Builds the BVH of the canonical primitives into `nodes` (bvh_node_capacity entries)
// and `leaf_prims` (3N float4).  scratch must hold bvh_scratch_bytes(N).  Returns 0 on
// success, else a cudaError_t value (or -1 when the builder's internal bounds were hit).
int bvh_build(const float *d_tri_v, int n_tris, const float4 *d_rects, const int *d_prim_flags, int n_rects,
              const float4 *d_spheres, int n_spheres, BvhNode *nodes, float4 *leaf_prims, void *scratch,
              cudaStream_t stream, BvhBuildInfo *info, std::function<void()> meanwhile, const int **pending) {
    *pending = nullptr;
    const int N = n_tris + n_rects + n_spheres;
    const size_t n = (size_t)(N > 0 ? N : 1);
    BuildArrays B;
    carve_build(B, (char *)scratch, N);
    int *kc = B.counters;
    const int max_nodes = bvh_node_capacity(N);
    const int grid_n = cdiv((long long)n, 256) < 148 * 8 ? cdiv((long long)n, 256) : 148 * 8;
    init_kernel<<<1, 32, 0, stream>>>(B.root_bounds, kc);
    prim_prepare_kernel<<<grid_n, 256, 0, stream>>>(d_tri_v, n_tris, d_rects, n_rects, d_spheres, d_prim_flags,
                                                    n_spheres, B.aabb_lo, B.aabb_hi, B.prims_canon, B.idx[0],
                                                    B.root_bounds);
    root_kernel<<<1, 1024, 0, stream>>>(B.root_bounds, N, nodes, B.tasks[0], B.cbs[0], B.small, B.mid, B.bins[0], B.chunks,
                                        B.task_first_chunk, kc);
    // a level halves its tasks at best; a task has more than SMALL_MAX primitives, so a level holds
    // at most N / SMALL_MAX of them.  SAH splits are uneven: four levels more than halving takes,
    // then as many as it needs, four at a time.
    int level = 0, until = 0, h[K_NUM] = {};
    if (N > SMALL_MAX) {
        until = 4;
        for (size_t m = n; m > SMALL_MAX; m >>= 1) ++until;
    }
    for (;;) {
        for (; level < until; ++level) {
            const int cur = level & 1;
            int *n_cur = kc + K_LARGE + cur, *n_next = kc + K_LARGE + (cur ^ 1);
            long long most = level < 30 ? 1LL << level : (long long)n;
            if (most > (long long)(n / SMALL_MAX) + 1) most = (long long)(n / SMALL_MAX) + 1;
            const int max_ch = (int)((long long)(n / CHUNK) + most + 1), warps = cdiv(most * 32, 128);
            bin_kernel<<<max_ch, BIN_THREADS, 0, stream>>>(B.chunks, kc + K_CHUNKS, B.idx[cur], B.aabb_lo, B.aabb_hi,
                                                           B.cbs[cur], B.bins[cur]);
            split_kernel<<<warps, 128, 0, stream>>>(B.tasks[cur], n_cur, B.bins[cur], B.bins[cur ^ 1],
                                                    (int)(n / SMALL_MAX + 2), B.child_bounds, B.dec);
            count_kernel<<<max_ch, BIN_THREADS, 0, stream>>>(B.chunks, kc + K_CHUNKS, B.tasks[cur], B.dec, B.idx[cur],
                                                             B.aabb_lo, B.aabb_hi, B.cbs[cur], B.chunk_left);
            chunk_scan_kernel<<<warps, 128, 0, stream>>>(B.chunks, kc + K_CHUNKS, n_cur, B.chunk_left, B.chunk_loff,
                                                         B.task_first_chunk, B.dec);
            scatter_kernel<<<max_ch, BIN_THREADS, 0, stream>>>(B.chunks, kc + K_CHUNKS, B.tasks[cur], B.dec, B.idx[cur],
                                                               B.idx[cur ^ 1], B.aabb_lo, B.aabb_hi, B.cbs[cur],
                                                               B.chunk_loff, B.child_bounds);
            level_kernel<<<1, 1024, 0, stream>>>(B.tasks[cur], n_cur, B.dec, B.child_bounds, N, max_nodes, nodes,
                                                 B.tasks[cur ^ 1], B.cbs[cur ^ 1], n_next, B.small, cur ^ 1, B.chunks,
                                                 B.task_first_chunk, kc);
        }
        // the small tasks found so far (all of them, unless the expected levels did not suffice)
        // resident blocks, fewer for few primitives; warps take tasks in turn
        const int small_grid = std::min(148 * 8, cdiv((long long)n, 32 * SMALL_WARPS));
        if (N > SMALL_MID)
            small_build_kernel<SMALL_MAX><<<small_grid, 32 * SMALL_WARPS, 0, stream>>>(
                B.small, kc + K_SMALL, h[K_SMALL], N, B.idx[0], B.idx[1], B.aabb_lo, B.aabb_hi, nodes, max_nodes, B.mid, kc);
        small_build_kernel<SMALL_MID><<<2 * small_grid, 32 * SMALL_WARPS, 0, stream>>>(
            B.mid, kc + K_MID, h[K_MID], N, B.idx[0], B.idx[1], B.aabb_lo, B.aabb_hi, nodes, max_nodes, nullptr, kc);
        if (meanwhile) meanwhile();
        meanwhile = nullptr;
        if (N <= BVH_DEFERRED) {
            *pending = kc;
            break;
        }
        cudaMemcpyAsync(h, kc, sizeof(h), cudaMemcpyDeviceToHost, stream);
        const cudaError_t e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return (int)e;
        if (h[K_ERR] || level > 80) return -1;
        if (h[K_LARGE + (level & 1)] == 0) break;
        until = level + 4;
    }
    gather_leaf_prims_kernel<<<grid_n, 256, 0, stream>>>(B.idx[0], N, B.prims_canon, leaf_prims);
    return *pending ? 0 : bvh_build_check(h, N, info);
}

int bvh_build_check(const int *h, int n_prims, BvhBuildInfo *info) {
    if (h[K_ERR]) return -1;
    if (info) {
        info->large_levels = h[K_LEVELS];
        info->small_tasks = h[K_SMALL];
        info->node_capacity = bvh_node_capacity(n_prims);
        info->node_high_water = PAIRS + 2 * (n_prims > 0 ? n_prims : 1) + 2 * h[K_SPARE];
    }
    return 0;
}

}  // namespace rumi
