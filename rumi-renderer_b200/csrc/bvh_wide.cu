// Collapse of the binary SAH tree into the four-wide tree (wide.cuh) that the default walk
// reads.
//
// Each four-wide node is made from one binary interior node: start from its two children and,
// while fewer than four, open the interior candidate of largest surface area (its two children
// take its place).  One launch per level of the four-wide tree, a thread per frontier node: it
// fills its node, allocates its interior children as one contiguous block after itself and
// appends them to the next frontier, and appends its leaves to a list of records to write.  The
// host does not wait between levels (a launch on an empty frontier costs about 2 us); it reads the
// counts once, then allocates the two arrays to size and writes the leaf records, a warp per
// leaf.
#include "renderer.h"
#include "traverse.cuh"

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

// level: this launch's frontier is in[0 .. k[K_LEVELS + level]), the next one's count goes to
// k[K_LEVELS + level + 1] (the counts start at zero, the first at one).
__global__ void collapse_level(const BvhNode *__restrict__ nodes2, int n_nodes2, const float4 *__restrict__ lp,
                               int n_prims, const Frontier *__restrict__ in, Frontier *__restrict__ out, int level,
                               WideNode *__restrict__ wide, LeafJob *__restrict__ jobs, int cap, int *__restrict__ kc) {
    const int n_in = kc[K_LEVELS + level];
    int *n_out = kc + K_LEVELS + level + 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in; i += gridDim.x * blockDim.x) {
        const Frontier f = in[i];
        if (f.b2 < 0 || f.b2 >= n_nodes2 || f.b4 < 0 || f.b4 >= cap) {
            atomicExch(kc + K_ERR, 1);
            return;
        }
        const BvhNode top = nodes2[0];
        const float amax = fmaxf(fmaxf(fmaxf(fabsf(top.lo_x), fabsf(top.hi_x)), fmaxf(fabsf(top.lo_y), fabsf(top.hi_y))),
                                 fmaxf(fabsf(top.lo_z), fabsf(top.hi_z)));
        const float pad = wide_pad(amax);
        int cand[4], kind[4];
        int nc = 0;
        const BvhNode root = nodes2[f.b2];
        const int rk = n_prims > 0 ? node_kind(root, n_nodes2) : 0;
        if (rk == 1) {
            cand[0] = f.b2;  // a leaf root: one leaf child
            kind[0] = 1;
            nc = 1;
        } else if (rk == 2) {
            for (int s = 0; s < 2; ++s) {
                const int k = node_kind(nodes2[root.first + s], n_nodes2);
                if (k) {
                    cand[nc] = root.first + s;
                    kind[nc] = k;
                    ++nc;
                }
            }
            // open the interior candidate of largest surface area while there is room
            while (nc < 4) {
                int best = -1;
                float best_a = -1.0f;
                for (int k = 0; k < nc; ++k) {
                    if (kind[k] != 2) continue;
                    const float a = half_area(nodes2[cand[k]]);
                    if (a > best_a) {
                        best_a = a;
                        best = k;
                    }
                }
                if (best < 0) break;
                const int first = nodes2[cand[best]].first;
                // remove `best`, append its usable children
                for (int k = best; k + 1 < nc; ++k) {
                    cand[k] = cand[k + 1];
                    kind[k] = kind[k + 1];
                }
                --nc;
                for (int s = 0; s < 2; ++s) {
                    const int k = node_kind(nodes2[first + s], n_nodes2);
                    if (k) {
                        cand[nc] = first + s;
                        kind[nc] = k;
                        ++nc;
                    }
                }
            }
        }
        int n_int = 0;
        for (int k = 0; k < nc; ++k) n_int += kind[k] == 2 ? 1 : 0;
        int base = 0, pos = 0;
        if (n_int > 0) {
            base = atomicAdd(kc + K_WIDE, n_int);
            pos = atomicAdd(n_out, n_int);
            // (the walk counts on children that come after their parent: it then ends)
            if (base + n_int > cap || base <= f.b4) {
                atomicExch(kc + K_ERR, 3);
                return;
            }
        }
        WideNode o;
        int j = 0;
        for (int k = 0; k < 4; ++k) {
            if (k >= nc) {
                wide_empty(o, k);
                continue;
            }
            const BvhNode c = nodes2[cand[k]];
            if (kind[k] == 1) {
                if (c.first < 0 || c.count > n_prims - c.first) {
                    atomicExch(kc + K_ERR, 4);
                    return;
                }
                const int nr = leaf_records(lp, c.first, c.count);
                const int at = atomicAdd(kc + K_RECS, nr);
                const int job = atomicAdd(kc + K_JOBS, 1);
                if (at + nr > n_prims + 1 || job >= n_prims) {
                    atomicExch(kc + K_ERR, 5);
                    return;
                }
                jobs[job] = LeafJob{c.first, c.count, at};
                wide_child(o, k, c, pad, ~at);
            } else {
                wide_child(o, k, c, pad, base + j);
                out[pos + j] = Frontier{cand[k], base + j};
                ++j;
            }
        }
        wide[f.b4] = o;
    }
}

// A warp per leaf: its triangles two by two in order, then its other primitives.
__global__ void records_kernel(const float4 *__restrict__ lp, const LeafJob *__restrict__ jobs, int n_jobs,
                               LeafRec *__restrict__ recs) {
    const int lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w == 0 && lane == 0) {  // record 0: nothing hits it
        LeafRec z = {};
        z.id[0] = REC_LAST;
        recs[0] = z;
    }
    if (w >= n_jobs) return;
    const LeafJob jb = jobs[w];
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

}  // namespace

// Builds the four-wide tree of a finished binary tree; *wide_out and *recs_out are allocated to
// size.  Returns 0, a cudaError_t value, or -1 when an index left its range.
int bvh_wide(const BvhNode *nodes2, int n_nodes2, const float4 *lp, int n_prims, WideNode **wide_out, int *n_wide,
             LeafRec **recs_out, int *n_recs, cudaStream_t stream) {
    // one four-wide node at most per leaf, one job per leaf: a node with an interior child has four
    // children, so nodes are outnumbered by leaves
    const size_t cap = n_prims > 1 ? (size_t)n_prims : 1;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_wide = al(cap * sizeof(WideNode)), b_front = al(cap * sizeof(Frontier)), b_jobs = al(cap * sizeof(LeafJob));
    char *tmp = nullptr;
    cudaError_t e = dalloc((void **)&tmp, b_wide + 2 * b_front + b_jobs + al(K_NUM * sizeof(int)), stream);
    if (e != cudaSuccess) return (int)e;
    WideNode *wide = (WideNode *)tmp;
    Frontier *fr[2] = {(Frontier *)(tmp + b_wide), (Frontier *)(tmp + b_wide + b_front)};
    LeafJob *jobs = (LeafJob *)(tmp + b_wide + 2 * b_front);
    int *kc = (int *)(tmp + b_wide + 2 * b_front + b_jobs);
    int h[K_NUM] = {};
    h[K_WIDE] = 1;
    h[K_RECS] = 1;  // record 0 is the one nothing hits
    h[K_LEVELS] = 1;
    const Frontier root{0, 0};
    cudaMemcpyAsync(kc, h, sizeof(h), cudaMemcpyHostToDevice, stream);
    cudaMemcpyAsync(fr[0], &root, sizeof(root), cudaMemcpyHostToDevice, stream);
    // levels are launched a few at a time past the expected depth (four-wide: half of log2), up to
    // the binary tree's deepest level
    int level = 0, expect = 2;
    for (size_t n = cap; n > 16; n >>= 2) ++expect;
    expect += expect / 4;
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
        cudaMemcpyAsync(h, kc, sizeof(h), cudaMemcpyDeviceToHost, stream);
        e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess || h[K_ERR] || h[K_LEVELS + level] == 0 || level >= 128) break;
        expect = level + 4;
    }
    WideNode *w = nullptr;
    LeafRec *r = nullptr;
    const bool ok = e == cudaSuccess && !h[K_ERR] && h[K_LEVELS + level] == 0;
    if (ok) e = dalloc((void **)&w, sizeof(WideNode) * (size_t)h[K_WIDE], stream);
    if (ok && e == cudaSuccess) e = dalloc((void **)&r, sizeof(LeafRec) * (size_t)h[K_RECS], stream);
    if (ok && e == cudaSuccess) {
        cudaMemcpyAsync(w, wide, sizeof(WideNode) * (size_t)h[K_WIDE], cudaMemcpyDeviceToDevice, stream);
        records_kernel<<<(h[K_JOBS] + 4) / 4, 128, 0, stream>>>(lp, jobs, h[K_JOBS], r);
        e = cudaGetLastError();
    }
    dfree(tmp, stream);
    if (!ok || e != cudaSuccess) {
        dfree(w, stream);
        dfree(r, stream);
        return e != cudaSuccess ? (int)e : -1;
    }
    *wide_out = w;
    *n_wide = h[K_WIDE];
    *recs_out = r;
    *n_recs = h[K_RECS];
    return 0;
}

}  // namespace rumi
