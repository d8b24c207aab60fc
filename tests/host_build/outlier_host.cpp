// The walk of walk_host.cpp with the primitives that it tests counted.  Test infrastructure, not
// part of the library.
#include "walk_host.cpp"

extern "C" {

// Arguments as rumi_host_walk's; returns the number of primitives tested by the walk of all rays.
int rumi_host_walk_tests(const float *prims, const float *boxes, int n, int seed, const float *rays, int n_rays) {
    Tree T;
    std::vector<float4> p(3 * (size_t)n);
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
    T.fill(0, 0, n);
    DevScene s;
    memset(&s, 0, sizeof(s));
    s.wide = (const float4 *)T.nodes.data();
    s.recs = (const float4 *)T.recs.data();
    static int stack[8 * WW_THREADS];
    int counter = 0;
    TraceStats st{0, 0};
    threadIdx.x = 0;
    traverse_queue_ww<false, 8, true, false>(
        [&](int) { return &s; }, n_rays, &counter, 1, stack,
        [&](int i, float3 &o, float3 &d, float &tmax, bool &in_obj) {
            const float *r = rays + 8 * i;
            o = mk3(r[0], r[1], r[2]);
            in_obj = r[3] != 0.0f;
            d = mk3(r[4], r[5], r[6]);
            tmax = r[7];
        },
        [&](int, const HitRec &) {}, st);
    return st.prims;
}

}  // extern "C"
