// The four-wide tree of the default walk: node and leaf-record formats and their packing
// (host and device, so that a host test builds the same bytes).
#pragma once
#include "common.cuh"
#include <cmath>

// 96-byte four-wide node (three 32-byte loads): four child boxes as centre and half extent.
// A word of hxy holds two half extents: as a float it is at least that of y (the lower bits only
// add to it), shifted up by 16 it is that of x, rounded up to 16 bits.  x and y of a centre are
// adjacent, so that one packed operation (fma.rn.f32x2) serves both axes with the ray's
// constants as they lie in registers, and with |1/d| per ray the slab ends are t_c -+ h |1/d|:
// no minimum or maximum picks near from far, which matters because those run at half the rate of
// multiply-adds.  The walk is bound by issue (65% active) with half of the lanes waiting, then by the
// L1's rate for divergent loads (one 128-byte line per cycle and SM: 73%; with a 128-byte node in four
// loads it was 80% and the first bound) and by the half-rate pipe (59%).  Measured per 1024x1024x64 frame of the 1M-triangle workload, closest-hit
// / any-hit: binary tree, scalar slabs 85.8 / 46.5 ms; binary, this slab form 78.5 / 42.1;
// four-wide with 32-bit half extents (128 bytes) 71.6 / 38.7; this node 64.1 / 33.9 (52.3 / 29.0 with
// the rays of a large wave in order); a 64-byte node with 8-bit planes 73.9 / 40.1 (the byte decoding
// costs more half-rate operations than the saved load is worth).
// ref[k] >= 0: node index of child k, larger than the node's own; ref[k] < 0: its leaf, whose
// records start at recs[~ref[k]].  An empty slot has negative half extents, which no ray with
// finite origin enters, and refers to record 0, which nothing hits.  wide[0] is the root.
struct __align__(32) WideNode {
    float2 cxy[4];
    float cz[4];
    unsigned hxy[4];
    float hz[4];
    int ref[4];
};
static_assert(sizeof(WideNode) == 96, "WideNode is three 32-byte loads");

// 96-byte leaf record: two triangles, every component of the pair adjacent (-v0, e1, e2 per axis)
// for the packed operations, or one rect or sphere as its three leaf_prims float4.  id[0] carries
// the flags; an odd triangle fills both places.
struct __align__(32) LeafRec {
    float nv[6], e1[6], e2[6];
    unsigned id[2];
    unsigned unused[4];
};
static_assert(sizeof(LeafRec) == 96, "LeafRec is three 32-byte loads");
#define REC_LAST 0x80000000u    // the leaf's last record
#define REC_SINGLE 0x40000000u  // a rect or sphere
#define REC_ID 0x3fffffffu

RUMI_HD unsigned wide_bits(float f) {
    union {
        float f;
        unsigned u;
    } v;
    v.f = f;
    return v.u;
}

// Absolute padding of child boxes in a scene whose largest coordinate is amax: 2^-21 of it
// exceeds the rounding of (c - o) / d and of o / d for origins within a few scene extents (the
// binary node's own padding is relative to each face).
RUMI_HD float wide_pad(float amax) { return amax * 4.76837158203125e-7f; }

// The part of it that the box c gets: no more than 1/128 of its largest extent, or 2^-20 of its
// largest coordinate where that is more.  One far primitive (a sky sphere, a ground plane, a stray
// vertex) would otherwise widen every box of the scene: a million triangles of 0.25 units inside a
// sphere of radius 10^4 rendered in 148 ms and inside one of 10^5 in 7.5 s, against 20 without it.
RUMI_HD float wide_box_pad(const BvhNode &c, float pad) {
    const float ext = fmaxf(fmaxf(c.hi_x - c.lo_x, c.hi_y - c.lo_y), c.hi_z - c.lo_z);
    const float far = fmaxf(fmaxf(fmaxf(fabsf(c.lo_x), fabsf(c.hi_x)), fmaxf(fabsf(c.lo_y), fabsf(c.hi_y))),
                            fmaxf(fabsf(c.lo_z), fabsf(c.hi_z)));
    return fminf(pad, fmaxf(0.0078125f * ext, 9.5367431640625e-7f * far));
}

// Half extent of [lo, hi] about c, padded, rounded up.
RUMI_HD float wide_half(float lo, float hi, float c, float pad) {
    const double up = (double)hi - c, dn = (double)c - lo;
    const double h = (up > dn ? up : dn) + pad;
    const float f = (float)h;
    return (double)f < h ? nextafterf(f, INFINITY) : f;
}

RUMI_HD void wide_set_half(WideNode &o, int k, float hx, float hy, float hz) {
    const unsigned x = (wide_bits(hx) + 0xffffu) >> 16, y = wide_bits(hy);
    // the smallest upper half with which the whole word is no smaller than hy
    o.hxy[k] = x | ((y & 0xffffu) > x ? (y & 0xffff0000u) + 0x10000u : y & 0xffff0000u);
    o.hz[k] = hz;
}

RUMI_HD void wide_empty(WideNode &o, int k) {
    o.cxy[k] = make_float2(0.0f, 0.0f);
    o.cz[k] = 0.0f;
    wide_set_half(o, k, -1e30f, -1e30f, -1e30f);
    o.ref[k] = ~0;
}

// Centre and half extent of [lo, hi].  An interval that reaches past 2^47 becomes +-2^126 about 0, which
// every ray is in: c |1/d| stays finite up to there (|1/d| <= 2^80, safe_rcp), and a centre that does
// not would put both ends of the slab at the same infinity, where its finite end may be entered.
RUMI_HD void wide_axis(float lo, float hi, float pad, float &c, float &h) {
    if (fabsf(lo) > 1.40737488e14f || fabsf(hi) > 1.40737488e14f) {
        c = 0.0f;
        h = 8.50705917e37f;
        return;
    }
    c = 0.5f * lo + 0.5f * hi;
    h = wide_half(lo, hi, c, pad);
}

// scene_pad: wide_pad of the scene.
RUMI_HD void wide_child(WideNode &o, int k, const BvhNode &c, float scene_pad, int ref) {
    const float pad = wide_box_pad(c, scene_pad);
    float hx, hy, hz;
    wide_axis(c.lo_x, c.hi_x, pad, o.cxy[k].x, hx);
    wide_axis(c.lo_y, c.hi_y, pad, o.cxy[k].y, hy);
    wide_axis(c.lo_z, c.hi_z, pad, o.cz[k], hz);
    wide_set_half(o, k, hx, hy, hz);
    o.ref[k] = ref;
}

// Triangle in place `slot` of a record, from its leaf_prims float4.
RUMI_HD void rec_triangle(LeafRec &r, int slot, float4 A, float4 B, float4 C) {
    r.nv[slot] = -A.x; r.nv[2 + slot] = -A.y; r.nv[4 + slot] = -A.z;
    r.e1[slot] = B.x; r.e1[2 + slot] = B.y; r.e1[4 + slot] = B.z;
    r.e2[slot] = C.x; r.e2[2 + slot] = C.y; r.e2[4 + slot] = C.z;
    r.id[slot] = wide_bits(A.w);
}

RUMI_HD void rec_single(LeafRec &r, float4 A, float4 B, float4 C) {
    float4 *f = reinterpret_cast<float4 *>(&r);
    f[0] = A;
    f[1] = B;
    f[2] = C;
    r.id[0] = wide_bits(A.w) | REC_SINGLE;
}

// A rect's record also holds what its test derives from the edges alone (the Rect constructor's
// values, which cost more than the rest of the test): normal, lengths, and the factors
// inv_area * width and inv_area * length.
RUMI_HD void rec_rect(LeafRec &r, float4 A, float4 B, float4 C, float3 n, float length, float width, float by_width,
                      float by_length) {
    float4 *f = reinterpret_cast<float4 *>(&r);
    f[3] = make_float4(n.x, n.y, n.z, length);
    f[4].x = width;
    f[4].y = by_width;
    f[5].x = by_length;
    rec_single(r, A, B, C);
}
