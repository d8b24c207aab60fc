// Collapse of the binary SAH tree into the four-wide tree (wide.cuh) that the default walk
// reads.
//
// Each four-wide node is made from one binary interior node: start from its two children and,
// while fewer than four, open the interior candidate of largest surface area (its two children
// take its place).  One launch per level of the four-wide tree, a thread per frontier node: it
// fills its node, allocates its interior children as one contiguous block after itself and
// appends them to the next frontier, and appends its leaves to a list of records to write, a warp per
// leaf.  The host does not wait between levels (a launch on an empty frontier costs about 2 us); it
// reads the counts once, then allocates the two arrays to size and writes the leaf records.  A small
// scene's tree is made by one block in one launch, in arrays for as many nodes and records as there
// can be: build and collapse are a chain of short launches and waits there, and a scene of 11 primitives
// is created in 0.25 ms, 0.31 with three launches, two copies and a wait for the levels (0.26 without
// this tree).
#include "renderer.h"
#include "traverse.cuh"
#include <algorithm>

namespace rumi {

namespace {

struct Frontier {
    int b2;  // binary node
    int b4;  // four-wide node to fill
};
struct LeafJob {
    int first, count;  // leaf_prims range
    int at;            // first record
};
enum { K_IN = 0, K_OUT = 1, K_WIDE = 2, K_RECS = 3, K_JOBS = 4, K_ERR = 5, K_LEVELS = 8, K_NUM = 8 + 130 };

__device__ __forceinline__ float half_area(const BvhNode &n) {
    const float dx = n.hi_x - n.lo_x, dy = n.hi_y - n.lo_y, dz = n.hi_z - n.lo_z;
    return dx * dy + dy * dz + dz * dx;
}

// 1: leaf, 2: interior with a usable child pair and a non-empty box, 0: nothing to keep
// (the binary builder leaves an empty side of a degenerate split as a count-0 node with
// an empty box and no children; the binary traversal never enters it, the collapse drops it).
__device__ __forceinline__ int node_kind(const BvhNode &c, int n_nodes2) {
    if (c.count > 0) return 1;
    if (c.count == 0 && c.first >= 2 && c.first + 1 < n_nodes2 && c.lo_x <= c.hi_x && c.lo_y <= c.hi_y &&
        c.lo_z <= c.hi_z)
        return 2;
    return 0;
}

// Records of the leaf [first, first + count): triangles two by two, any other primitive alone.
__device__ __forceinline__ int leaf_records(const float4 *__restrict__ lp, int first, int count) {
    int tris = 0;
    for (int i = first; i < first + count; ++i) {
        const int tag = __float_as_int(__ldg(&lp[3 * (size_t)i + 1].w));
        tris += (tag & 0xff) == PRIM_TRI ? 1 : 0;
    }
    return (tris + 1) / 2 + (count - tris);
}

// Adds every lane's v to *counter with one addition (additions to one address are serial); returns
// the sum before the lane's own.
__device__ __forceinline__ int warp_add(int *counter, int v) {
    const int lane = threadIdx.x & 31;
    int incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    int base = 0;
    if (lane == 31 && incl > 0) base = atomicAdd(counter, incl);
    return __shfl_sync(0xffffffffu, base, 31) + incl - v;
}

// A four-wide node's children being chosen: binary nodes, interior (kind 2) or leaf (1).
struct Candidates {
    int node[4], kind[4], n;
    float area[4];  // of the interior ones
    BvhNode box[4];

    __device__ void add(const BvhNode *__restrict__ nodes2, int n_nodes2, int i) {
        const BvhNode b = nodes2[i];
        const int k = node_kind(b, n_nodes2);
        if (!k) return;
#pragma unroll
        for (int s = 0; s < 4; ++s)
            if (s == n) {
                node[s] = i;
                kind[s] = k;
                area[s] = k == 2 ? half_area(b) : -1.0f;
                box[s] = b;
            }
        ++n;
    }
    // the children of the interior candidate of largest surface area in its place; false: none
    __device__ bool open(const BvhNode *__restrict__ nodes2, int n_nodes2) {
        float best = -1.0f;
        int at = -1, first = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < n && kind[k] == 2 && area[k] > best) {
                best = area[k];
                at = k;
                first = box[k].first;
            }
        if (at < 0) return false;
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (k >= at && k + 1 < n) {
                node[k] = node[k + 1];
                kind[k] = kind[k + 1];
                area[k] = area[k + 1];
                box[k] = box[k + 1];
            }
        --n;
        add(nodes2, n_nodes2, first);
        add(nodes2, n_nodes2, first + 1);
        return true;
    }
};

// Fills the four-wide nodes of the frontier in[0 .. n_in) (in == nullptr: the root alone) and appends
// their interior children to out; thread `first` of `stride`.  A level lasts as long as its serial
// parts: the additions to the four counters, so a warp makes one of each, and the chain of node loads,
// so candidates stay in registers with their boxes (a million triangles: build and collapse
// 3.37 -> 3.16 ms).  All counts start at zero: the nodes are counted without the root, the records
// without the empty one.
__device__ __forceinline__ void collapse_front(const BvhNode *__restrict__ nodes2, int n_nodes2,
                                               const float4 *__restrict__ lp, int n_prims,
                                               const Frontier *in, int n_in, Frontier *out, int *n_out, WideNode *wide,
                                               LeafJob *jobs, int cap, int *kc, int first, int stride) {
    const BvhNode top = nodes2[0];
    const float amax = fmaxf(fmaxf(fmaxf(fabsf(top.lo_x), fabsf(top.hi_x)), fmaxf(fabsf(top.lo_y), fabsf(top.hi_y))),
                             fmaxf(fabsf(top.lo_z), fabsf(top.hi_z)));
    const float pad = wide_pad(amax);
    const int lane = threadIdx.x & 31;
    for (int i = first; i - lane < n_in; i += stride) {
        const Frontier f = i < n_in && in ? in[i] : Frontier{0, 0};
        int err = f.b2 < 0 || f.b2 >= n_nodes2 || f.b4 < 0 || f.b4 >= cap ? 1 : 0;
        Candidates c;
        c.n = 0;
        if (i < n_in && !err && n_prims > 0) {
            const BvhNode root = nodes2[f.b2];
            const int rk = node_kind(root, n_nodes2);
            if (rk == 1) {
                c.add(nodes2, n_nodes2, f.b2);  // a leaf root: one leaf child
            } else if (rk == 2) {
                c.add(nodes2, n_nodes2, root.first);
                c.add(nodes2, n_nodes2, root.first + 1);
                // open the interior candidate of largest surface area while there is room
                while (c.n < 4 && c.open(nodes2, n_nodes2)) {}
            }
        }
        int n_int = 0, n_leaf = 0, nr[4], n_rec = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            nr[k] = 0;
            if (k >= c.n) continue;
            if (c.kind[k] == 2) {
                ++n_int;
            } else if (c.box[k].first < 0 || c.box[k].count > n_prims - c.box[k].first) {
                err = 4;
            } else {
                nr[k] = leaf_records(lp, c.box[k].first, c.box[k].count);
                n_rec += nr[k];
                ++n_leaf;
            }
        }
        if (err) n_int = n_leaf = n_rec = 0;
        const int base = 1 + warp_add(kc + K_WIDE, n_int), pos = warp_add(n_out, n_int);
        int at = 1 + warp_add(kc + K_RECS, n_rec), job = warp_add(kc + K_JOBS, n_leaf);
        // (the walk counts on children that come after their parent: it then ends)
        if (!err && n_int > 0 && (base + n_int > cap || base <= f.b4)) err = 3;
        if (!err && n_leaf > 0 && (at + n_rec > n_prims + 1 || job + n_leaf > n_prims)) err = 5;
        if (err) atomicExch(kc + K_ERR, err);
        if (err || i >= n_in) continue;
        WideNode o;
        int j = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= c.n) {
                wide_empty(o, k);
            } else if (c.kind[k] == 1) {
                jobs[job++] = LeafJob{c.box[k].first, c.box[k].count, at};
                wide_child(o, k, c.box[k], pad, ~at);
                at += nr[k];
            } else {
                wide_child(o, k, c.box[k], pad, base + j);
                out[pos + j] = Frontier{c.node[k], base + j};
                ++j;
            }
        }
        wide[f.b4] = o;
    }
}

// One level of a large tree: the frontier is in[0 .. kc[K_LEVELS + level]), the next one's count goes
// to kc[K_LEVELS + level + 1].
__global__ void collapse_level(const BvhNode *__restrict__ nodes2, int n_nodes2, const float4 *__restrict__ lp,
                               int n_prims, const Frontier *__restrict__ in, Frontier *__restrict__ out, int level,
                               WideNode *__restrict__ wide, LeafJob *__restrict__ jobs, int cap, int *__restrict__ kc) {
    collapse_front(nodes2, n_nodes2, lp, n_prims, level > 0 ? in : nullptr, level > 0 ? kc[K_LEVELS + level] : 1, out,
                   kc + K_LEVELS + level + 1, wide, jobs, cap, kc, blockIdx.x * blockDim.x + threadIdx.x,
                   gridDim.x * blockDim.x);
}

// The records of one leaf, by a warp: its triangles two by two in order, then its other primitives.
__device__ __forceinline__ void leaf_job(const float4 *__restrict__ lp, const LeafJob &jb, LeafRec *recs) {
    const int lane = threadIdx.x & 31;
    auto is_tri = [&](int i) { return (__float_as_int(lp[3 * (size_t)(jb.first + i) + 1].w) & 0xff) == PRIM_TRI; };
    int n_tri = 0;
    for (int b = 0; b < jb.count; b += 32)
        n_tri += __popc(__ballot_sync(0xffffffffu, b + lane < jb.count && is_tri(b + lane)));
    const int pairs = (n_tri + 1) / 2, total = pairs + jb.count - n_tri;
    int tri0 = 0, one0 = 0;  // triangles / others before this batch of 32
    for (int b = 0; b < jb.count; b += 32) {
        const bool here = b + lane < jb.count;
        const bool tri = here && is_tri(b + lane);
        const unsigned mt = __ballot_sync(0xffffffffu, tri), mo = __ballot_sync(0xffffffffu, here && !tri);
        const unsigned lt = (1u << lane) - 1u;
        if (here) {
            const size_t q = 3 * (size_t)(jb.first + b + lane);
            const float4 A = lp[q], B = lp[q + 1], C = lp[q + 2];
            if (tri) {
                const int rank = tri0 + __popc(mt & lt), r = rank >> 1;
                LeafRec &rec = recs[jb.at + r];
                rec_triangle(rec, rank & 1, A, B, C);
                if (rank + 1 == n_tri && !(rank & 1)) rec_triangle(rec, 1, A, B, C);
                if (!(rank & 1) && r + 1 == total) rec.id[0] |= REC_LAST;
            } else {
                const int r = pairs + one0 + __popc(mo & lt);
                LeafRec &rec = recs[jb.at + r];
                if ((__float_as_int(B.w) & 0xff) == PRIM_RECT) {
                    const RectGeom g = rect_geom(f4xyz(B), f4xyz(C));
                    rec_rect(rec, A, B, C, g.n, g.length, g.width, __fmul_rn(g.inv_area, g.width),
                             __fmul_rn(g.inv_area, g.length));
                } else {
                    rec_single(rec, A, B, C);
                }
                if (r + 1 == total) rec.id[0] |= REC_LAST;
            }
        }
        tri0 += __popc(mt);
        one0 += __popc(mo);
    }
}

__device__ __forceinline__ void empty_record(LeafRec *recs) {  // record 0: nothing hits it
    LeafRec z = {};
    z.id[0] = REC_LAST;
    recs[0] = z;
}

__global__ void records_kernel(const float4 *__restrict__ lp, const LeafJob *__restrict__ jobs, int n_jobs,
                               LeafRec *__restrict__ recs) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w == 0 && (threadIdx.x & 31) == 0) empty_record(recs);
    if (w < n_jobs) leaf_job(lp, jobs[w], recs);
}

// The whole tree of a small scene by one block, counters in shared memory; they and the build's go to
// kc for the host.
static constexpr int SMALL_THREADS = 512;
__global__ void __launch_bounds__(SMALL_THREADS)
    collapse_small(const BvhNode *__restrict__ nodes2, int n_nodes2, const float4 *__restrict__ lp, int n_prims,
                   Frontier *fr0, Frontier *fr1, WideNode *wide, LeafJob *jobs, int cap, LeafRec *recs,
                   const int *build_kc, int *kc) {
    __shared__ int s_k[K_NUM];
    for (int k = threadIdx.x; k < K_NUM; k += SMALL_THREADS) s_k[k] = 0;
    __syncthreads();
    for (int level = 0; level < 128; ++level) {
        const int n_in = level > 0 ? s_k[K_LEVELS + level] : 1;
        if (n_in == 0) break;
        collapse_front(nodes2, n_nodes2, lp, n_prims, level == 0 ? nullptr : level & 1 ? fr1 : fr0, n_in,
                       level & 1 ? fr0 : fr1, s_k + K_LEVELS + level + 1, wide, jobs, cap, s_k, threadIdx.x, SMALL_THREADS);
        __syncthreads();
    }
    if (threadIdx.x == 0) empty_record(recs);
    if (!s_k[K_ERR])  // (else the jobs may have gaps)
        for (int w = threadIdx.x >> 5; w < s_k[K_JOBS]; w += SMALL_THREADS / 32) leaf_job(lp, jobs[w], recs);
    for (int k = threadIdx.x; k < K_NUM; k += SMALL_THREADS) kc[k] = s_k[k];
    if (threadIdx.x < BVH_COUNTERS) kc[K_NUM + threadIdx.x] = build_kc ? build_kc[threadIdx.x] : 0;
}

}  // namespace

// Builds the four-wide tree of a finished binary tree; *wide_out and *recs_out are allocated.  Of a
// small scene (BVH_DEFERRED) the build's counters, still on the device, are read with this tree's:
// build_kc to build_h.  Returns 0, a cudaError_t value, or -1 when an index left its range.
int bvh_wide(const BvhNode *nodes2, int n_nodes2, const float4 *lp, int n_prims, const int *build_kc, int *build_h,
             WideNode **wide_out, int *n_wide, LeafRec **recs_out, int *n_recs, cudaStream_t stream) {
    // one four-wide node at most per leaf, one job per leaf: a node with an interior child has four
    // children, so nodes are outnumbered by leaves
    const size_t cap = n_prims > 1 ? (size_t)n_prims : 1;
    const bool small = n_prims <= BVH_DEFERRED;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_wide = small ? 0 : al(cap * sizeof(WideNode)), b_front = al(cap * sizeof(Frontier)),
                 b_jobs = al(cap * sizeof(LeafJob));
    WideNode *w = nullptr;
    LeafRec *r = nullptr;
    char *tmp = nullptr;
    cudaError_t e = dalloc((void **)&tmp, b_wide + 2 * b_front + b_jobs + al((K_NUM + BVH_COUNTERS) * sizeof(int)), stream);
    if (small && e == cudaSuccess) e = dalloc((void **)&w, sizeof(WideNode) * cap, stream);
    if (small && e == cudaSuccess) e = dalloc((void **)&r, sizeof(LeafRec) * (cap + 1), stream);
    if (e != cudaSuccess) {
        dfree(tmp, stream);
        dfree(w, stream);
        return (int)e;
    }
    WideNode *wide = small ? w : (WideNode *)tmp;
    Frontier *fr[2] = {(Frontier *)(tmp + b_wide), (Frontier *)(tmp + b_wide + b_front)};
    LeafJob *jobs = (LeafJob *)(tmp + b_wide + 2 * b_front);
    int *kc = (int *)(tmp + b_wide + 2 * b_front + b_jobs);
    int h[K_NUM + BVH_COUNTERS] = {}, level = 0;
    if (small) {
        collapse_small<<<1, SMALL_THREADS, 0, stream>>>(nodes2, n_nodes2, lp, n_prims, fr[0], fr[1], wide, jobs, (int)cap,
                                                        r, build_kc, kc);
        cudaMemcpyAsync(h, kc, sizeof(h), cudaMemcpyDeviceToHost, stream);
        e = cudaStreamSynchronize(stream);
        level = 128;
        if (build_h) std::copy(h + K_NUM, h + K_NUM + BVH_COUNTERS, build_h);
    } else {
        cudaMemsetAsync(kc, 0, K_NUM * sizeof(int), stream);
        // levels are launched a few at a time past the expected depth (four-wide: half of log2), up to
        // the binary tree's deepest level
        int expect = 2;
        for (size_t n = cap; n > 16; n >>= 2) ++expect;
        expect += expect / 2;
        for (;;) {
            for (; level < expect && level < 128; ++level) {
                size_t most = 1;  // of a frontier at this level
                for (int k = 0; k < level && most < cap; ++k) most *= 4;
                if (most > cap) most = cap;
                const int grid = (int)((most + 63) / 64);
                collapse_level<<<grid < 1184 ? grid : 1184, 64, 0, stream>>>(nodes2, n_nodes2, lp, n_prims, fr[level & 1],
                                                                             fr[(level & 1) ^ 1], level, wide, jobs,
                                                                             (int)cap, kc);
            }
            cudaMemcpyAsync(h, kc, K_NUM * sizeof(int), cudaMemcpyDeviceToHost, stream);
            e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess || h[K_ERR] || h[K_LEVELS + level] == 0 || level >= 128) break;
            expect = level + 4;
        }
    }
    const bool ok = e == cudaSuccess && !h[K_ERR] && h[K_LEVELS + level] == 0;
    const int nodes = h[K_WIDE] + 1, records = h[K_RECS] + 1;
    if (ok && !small) {
        e = dalloc((void **)&w, sizeof(WideNode) * (size_t)nodes, stream);
        if (e == cudaSuccess) e = dalloc((void **)&r, sizeof(LeafRec) * (size_t)records, stream);
        if (e == cudaSuccess) {
            cudaMemcpyAsync(w, wide, sizeof(WideNode) * (size_t)nodes, cudaMemcpyDeviceToDevice, stream);
            records_kernel<<<(h[K_JOBS] + 4) / 4, 128, 0, stream>>>(lp, jobs, h[K_JOBS], r);
            e = cudaGetLastError();
        }
    }
    dfree(tmp, stream);
    if (!ok || e != cudaSuccess) {
        dfree(w, stream);
        dfree(r, stream);
        return e != cudaSuccess ? (int)e : -1;
    }
    *wide_out = w;
    *n_wide = nodes;
    *recs_out = r;
    *n_recs = records;
    return 0;
}

}  // namespace rumi
