// Host build of the default walk (traverse_queue_ww, traverse.cuh) over a four-wide tree packed
// by the library's own packing (wide.cuh): a random tree over the caller's primitives, walked
// by a warp of one lane, against a test of every primitive.  Test infrastructure, not part of
// the library.
#include "cuda_host_shim.h"
#include "../../rumi-renderer_b200/csrc/traverse.cuh"

#include <algorithm>
#include <random>
#include <vector>

namespace {

struct Box {
    float lo[3], hi[3];
};

struct Tree {
    std::vector<WideNode> nodes;
    std::vector<LeafRec> recs;
    const float4 *prims;
    const Box *boxes;
    std::vector<int> order;
    float pad;
    std::mt19937 rng;

    BvhNode bounds(int first, int count) const {  // with the builder's padding (pad_bounds)
        float lo[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, hi[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
        for (int i = first; i < first + count; ++i)
            for (int a = 0; a < 3; ++a) {
                lo[a] = std::min(lo[a], boxes[order[i]].lo[a]);
                hi[a] = std::max(hi[a], boxes[order[i]].hi[a]);
            }
        for (int a = 0; a < 3; ++a) {
            const float e = std::max(std::fabs(lo[a]), std::fabs(hi[a])) * 9.5367431640625e-7f + 1e-30f;
            lo[a] -= e;
            hi[a] += e;
        }
        return BvhNode{lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], first, count};
    }

    int leaf(int first, int count) {
        const int at = (int)recs.size();
        int held = -1;
        std::vector<int> one;
        auto add = [&](int a, int b) {
            LeafRec r = {};
            rec_triangle(r, 0, prims[3 * a], prims[3 * a + 1], prims[3 * a + 2]);
            rec_triangle(r, 1, prims[3 * b], prims[3 * b + 1], prims[3 * b + 2]);
            recs.push_back(r);
        };
        for (int i = first; i < first + count; ++i) {
            const int p = order[i];
            if ((__float_as_int(prims[3 * p + 1].w) & 0xff) != PRIM_TRI) {
                one.push_back(p);
            } else if (held < 0) {
                held = p;
            } else {
                add(held, p);
                held = -1;
            }
        }
        if (held >= 0) add(held, held);
        for (int p : one) {
            LeafRec r = {};
            const float4 A = prims[3 * p], B = prims[3 * p + 1], C = prims[3 * p + 2];
            if ((__float_as_int(B.w) & 0xff) == PRIM_RECT) {
                const RectGeom g = rect_geom(f4xyz(B), f4xyz(C));
                rec_rect(r, A, B, C, g.n, g.length, g.width, g.inv_area * g.width, g.inv_area * g.length);
            } else {
                rec_single(r, A, B, C);
            }
            recs.push_back(r);
        }
        recs.back().id[0] |= REC_LAST;
        return ~at;
    }

    void fill(int node, int first, int count) {
        const int ways = count == 1 ? 1 : 1 + (int)(rng() % std::min(4, count));
        std::vector<int> cut = {first, first + count};
        for (int k = 1; k < ways; ++k) cut.push_back(first + 1 + (int)(rng() % (count - 1)));
        std::sort(cut.begin(), cut.end());
        WideNode o;
        std::vector<std::pair<int, std::pair<int, int>>> todo;
        int k = 0;
        for (size_t j = 0; j + 1 < cut.size(); ++j) {
            const int n = cut[j + 1] - cut[j];
            if (n == 0) continue;
            const BvhNode b = bounds(cut[j], n);
            int ref;
            if (n == 1 || n == count || (n <= 16 && rng() % 2)) {
                ref = leaf(cut[j], n);
            } else {
                ref = (int)nodes.size();
                nodes.push_back(WideNode());
                todo.push_back({ref, {cut[j], n}});
            }
            wide_child(o, k++, b, pad, ref);
        }
        for (; k < 4; ++k) wide_empty(o, k);
        nodes[node] = o;
        for (auto &t : todo) fill(t.first, t.second.first, t.second.second);
    }
};

template <bool ANYHIT>
void walk(const DevScene &s, const float *rays, int n, float *t, int *id, float *uv) {
    static int stack[8 * WW_THREADS];  // 8 entries in the fast part: deep walks move some out
    int counter = 0;
    TraceStats st{0, 0};
    threadIdx.x = 0;
    traverse_queue_ww<ANYHIT, 8, false, false>(
        [&](int) { return &s; }, n, &counter, 1, stack,
        [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
            const float *r = rays + 8 * i;
            o = mk3(r[0], r[1], r[2]);
            in_obj = r[3] != 0.0f;
            d = mk3(r[4], r[5], r[6]);
            tmax = r[7];
        },
        [&](int i, const HitRec &h) {
            t[i] = h.t;
            id[i] = h.t > 0.0f ? h.id * 2 + h.back : -1;
            uv[2 * i] = h.u;
            uv[2 * i + 1] = h.v;
        },
        st);
}

}  // namespace

extern "C" {

// prims: n * 12 floats (leaf_prims records), boxes: n * 6 floats, rays: n_rays * 8 floats.  The
// results of the walk in t / id / uv (id doubled plus the back-face bit, -1 for a miss), those of
// a test of every primitive in t2 / id2 / uv2.
void rumi_host_walk(const float *prims, const float *boxes, int n, int seed, const float *rays, int n_rays, int anyhit,
                    float *t, int *id, float *uv, float *t2, int *id2, float *uv2) {
    Tree T;
    std::vector<float4> p(3 * (size_t)std::max(n, 1));
    memcpy(p.data(), prims, sizeof(float4) * 3 * (size_t)n);
    T.prims = p.data();
    T.boxes = (const Box *)boxes;
    T.rng.seed((unsigned)seed);
    for (int i = 0; i < n; ++i) T.order.push_back(i);
    std::sort(T.order.begin(), T.order.end(), [&](int a, int b) { return T.boxes[a].lo[0] < T.boxes[b].lo[0]; });
    float amax = 0.0f;
    for (int i = 0; i < 6 * n; ++i) amax = std::max(amax, std::fabs(boxes[i]));
    T.pad = wide_pad(amax);
    LeafRec z = {};
    z.id[0] = REC_LAST;
    T.recs.push_back(z);
    T.nodes.push_back(WideNode());
    if (n > 0)
        T.fill(0, 0, n);
    else
        for (int k = 0; k < 4; ++k) wide_empty(T.nodes[0], k);
    DevScene s;
    memset(&s, 0, sizeof(s));
    s.wide = (const float4 *)T.nodes.data();
    s.recs = (const float4 *)T.recs.data();
    s.leaf_prims = p.data();
    s.n_prims = n;
    if (anyhit)
        walk<true>(s, rays, n_rays, t, id, uv);
    else
        walk<false>(s, rays, n_rays, t, id, uv);
    for (int i = 0; i < n_rays; ++i) {
        const float *r = rays + 8 * i;
        HitRec h;
        h.t = 0.0f;
        h.id = -1;
        h.u = h.v = 0.0f;
        h.back = 0;
        TraceStats st{0, 0};
        const float3 o = mk3(r[0], r[1], r[2]), d = mk3(r[4], r[5], r[6]);
        if (d.x != 0.0f || d.y != 0.0f || d.z != 0.0f) {
            if (anyhit)
                leaf_isect<true, false>(s, 0, n, o, d, r[7], r[3] != 0.0f, h, st);
            else
                leaf_isect<false, false>(s, 0, n, o, d, r[7], r[3] != 0.0f, h, st);
        }
        t2[i] = h.t;
        id2[i] = h.t > 0.0f ? h.id * 2 + h.back : -1;
        uv2[2 * i] = h.u;
        uv2[2 * i + 1] = h.v;
    }
}

}  // extern "C"
