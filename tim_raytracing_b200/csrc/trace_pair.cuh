// trace_pair.cuh -- closest-hit rays on the reference's binary tree, both child boxes
// of a node in one 112-byte record.
//
// The walk is that of trace_plain.cuh: the same node order (child 1 first iff
// d1 < d0, the other child pushed), the same leaf order, the same triangle test, so
// the order-dependent closest-hit rule gives the reference's answer. What differs is
// the record (built by bvh_four.cu), which drops the minimum and maximum a slab test
// takes per axis and box and the per-node leaf record:
//   per axis, 2 x float4: (lo[2], hi[2]) (hi[2], lo[2]), one word per child
//   ref[2]      the record of an inner child's children, or a leaf as
//               bit 31 | triangles << 27 | first triangle (triangles 0: more than 15, or
//               none where all bits of the first triangle are set)
//   8 B         unused
// A pair of children l, l + 1 is stored at index l / 2: pairs are disjoint, so no two
// share one. A ray reads its near and far planes of an axis with one 16-byte load,
// from the first vector where its direction is positive, else from the second.
//
// Decisions. A slab value is t' = RN(RN(p - o) * inv), inv within 2u of 1/d
// (u = 2^-24), the reference's t = RN(RN(p - o) / d): for components of 0 or within
// [2^-100, 2^100] they differ by at most 5u |t'| + 2^-148, or both exceed 2^126 with
// the same sign, and for a zero component both are the same infinity, or NaN, which
// the maxima and minima here pass on so that no test below holds. With e = 2^-18:
//   RN(T' (1 - e) - tmin') >  tiny  ->  the box is hit  (tiny = 2^-100)
//   RN(T' (1 + e) - tmin') < -tiny  ->  it is missed
//   the larger of child 0's entry distances < -tiny, or RN(d0' (1 + e) - d1') < -tiny
//                                   ->  child 0 first; the latter mirrored, child 1
// (e and tiny exceed four times the error of the values and of the tests). Entries
// set by planes both children share are equal in the reference too: child 0 first.
// Anything else is decided by the reference's divisions (pair_exact). A ray
// outside the ranges has tiny = +inf and takes them at every node.
#pragma once
#include "common.cuh"
#include "trace_plain.cuh"
#include "trace_any.cuh"

namespace timrt {

constexpr float kPairUp = 1.0f + 3.814697265625e-06f, kPairDown = 1.0f - 3.814697265625e-06f;   // 1 +- 2^-18

__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void pair_init(const SceneView& s, TravState& st, uint32_t bottom) {
    st.ix = rcp_fast(st.r.dx);
    st.iy = rcp_fast(st.r.dy);
    st.iz = rcp_fast(st.r.dz);
    st.boxabs = (box_dir_ok(st.r.dx) && box_dir_ok(st.r.dy) && box_dir_ok(st.r.dz) && st.t <= 1.2676506002282294e30f)
                    ? 7.888609052210118e-31f   // 2^-100
                    : __int_as_float(0x7F800000);
    const char* base = reinterpret_cast<const char*>(s.pairs);
    st.px = base + (__float_as_uint(st.r.dx) >> 31 << 4);
    st.py = base + 32u + (__float_as_uint(st.r.dy) >> 31 << 4);
    st.pz = base + 64u + (__float_as_uint(st.r.dz) >> 31 << 4);
    st.refs = base + 96u;
    st.top = bottom;
    st.hit = false;
    st.node = s.root_pair;
}

// The references of record 0.
__device__ __forceinline__ const char* pair_refs(const SceneView& s) { return reinterpret_cast<const char*>(s.pairs) + 96u; }

// The slab values of one axis of both children.
__device__ __forceinline__ void pair_slab(float2 p, float o, float inv, float& t0, float& t1) {
    unpack2f(mul2(sub2(pack2f(p.x, p.y), pack2f(o, o)), pack2f(inv, inv)), t0, t1);
}

// What the margins leave open: equal entries by shared planes, or the reference's divisions.
struct PairOpen { bool h0, h1, first1; };
static __device__ __noinline__ PairOpen pair_exact(Ray r, float2 nx, float2 fx, float2 ny, float2 fy, float2 nz, float2 fz,
                                                   float tmax) {
    const float d0 = collide_box(r, nx.x, ny.x, nz.x, fx.x, fy.x, fz.x, tmax);
    const float d1 = collide_box(r, nx.y, ny.y, nz.y, fx.y, fy.y, fz.y, tmax);
    return {d0 >= 0.0f, d1 >= 0.0f, d1 < d0};
}

// One advance of one lane from record st.node (see plain_advance).
template <int BLOCK>
__device__ __forceinline__ void pair_advance(TravState& st, const char* refs, const uint32_t* dir) {
    const uint64_t off = (uint64_t)st.node * kPairBytes;
    const float4 X = __ldg(reinterpret_cast<const float4*>(st.px + off));
    const float4 Y = __ldg(reinterpret_cast<const float4*>(st.py + off));
    const float4 Z = __ldg(reinterpret_cast<const float4*>(st.pz + off));
    const uint2 ref = __ldg(reinterpret_cast<const uint2*>(refs + off));
    const uint32_t r0 = ref.x, r1 = ref.y;
    const float2 nx = make_float2(X.x, X.y), fx = make_float2(X.z, X.w);
    const float2 ny = make_float2(Y.x, Y.y), fy = make_float2(Y.z, Y.w);
    const float2 nz = make_float2(Z.x, Z.y), fz = make_float2(Z.z, Z.w);
    float ax0, ax1, ay0, ay1, az0, az1, bx0, bx1, by0, by1, bz0, bz1;
    pair_slab(nx, st.r.ox, st.ix, ax0, ax1);
    pair_slab(ny, st.r.oy, st.iy, ay0, ay1);
    pair_slab(nz, st.r.oz, st.iz, az0, az1);
    pair_slab(fx, st.r.ox, st.ix, bx0, bx1);
    pair_slab(fy, st.r.oy, st.iy, by0, by1);
    pair_slab(fz, st.r.oz, st.iz, bz0, bz1);
    const float u0 = max3_nan(ax0, ay0, az0), u1 = max3_nan(ax1, ay1, az1);
    const float n0 = max_nan(u0, 0.0f), n1 = max_nan(u1, 0.0f);
    const float T0 = min3_nan(min_nan(bx0, by0), bz0, st.t), T1 = min3_nan(min_nan(bx1, by1), bz1, st.t);
    const float tiny = st.boxabs;
    bool h0 = __fmaf_rn(T0, kPairDown, -n0) > tiny, h1 = __fmaf_rn(T1, kPairDown, -n1) > tiny;
    const bool m0 = __fmaf_rn(T0, kPairUp, -n0) < -tiny, m1 = __fmaf_rn(T1, kPairUp, -n1) < -tiny;
    const bool f0 = u0 < -tiny || __fmaf_rn(n0, kPairUp, -n1) < -tiny;
    bool first1 = __fmaf_rn(n1, kPairUp, -n0) < -tiny;
    const bool order = f0 || first1 || !(h0 && h1);
    if (!((h0 || m0) && (h1 || m1) && order)) {
        // hit both, entries within the margin: equal if every axis that could set one has the same plane
        const float lo = fminf(n0, n1);
        const bool same = (h0 && h1) && (nx.x == nx.y || __fmaf_rn(fmaxf(ax0, ax1), kPairUp, -lo) < -tiny) &&
                          (ny.x == ny.y || __fmaf_rn(fmaxf(ay0, ay1), kPairUp, -lo) < -tiny) &&
                          (nz.x == nz.y || __fmaf_rn(fmaxf(az0, az1), kPairUp, -lo) < -tiny);
        if (!same) {
            Ray r{st.r.ox, st.r.oy, st.r.oz, 0.f, 0.f, 0.f};
            get3<BLOCK>(dir, r.dx, r.dy, r.dz);
            const PairOpen q = pair_exact(r, nx, fx, ny, fy, nz, fz, st.t);
            h0 = q.h0;
            h1 = q.h1;
            first1 = q.first1;
        }
    }
    const bool both = h0 && h1;
    const bool take1 = both ? first1 : h1;
    stack_push<BLOCK>(st.top, first1 ? r0 : r1, both);
    if (h0 || h1) st.node = take1 ? r1 : r0;
    else st.node = stack_pop<BLOCK>(st.top);
}

// The outputs of a ray whose walk is over: the hit triangle's record words, its leaf's
// id and its barycentrics (the test's values once more) where they are asked for.
__device__ __forceinline__ void pair_finish(const SceneView& s, TravState& st, bool want_nid, bool want_bary) {
    st.rec0 = st.rec1 = st.rec2 = 0u;
    st.u = st.v = 0.0f;
    if (!st.hit) {
        st.nid = 0xFFFFFFFFu;
        return;
    }
    const uint32_t tri = st.nid;
    const float4* tp = s.ptris + 3u * tri;
    const float4 A = __ldg(tp), B = __ldg(tp + 1), C = __ldg(tp + 2);
    st.rec0 = __float_as_uint(A.w);
    st.rec1 = __float_as_uint(B.w);
    st.rec2 = __float_as_uint(C.w);
    if (want_bary)
        collide_triangle_e(st.r, A.x, A.y, A.z, B.x, B.y, B.z, C.x, C.y, C.z, __int_as_float(0x7F800000), st.u, st.v);
    if (want_nid) st.nid = __ldg(s.leaf4 + 2u * __ldg(s.tri_leaf4 + tri)).w;
}

}  // namespace timrt
