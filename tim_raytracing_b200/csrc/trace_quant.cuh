// trace_quant.cuh -- rays of one kind on the 8-wide quantised tree (trace_wide.cuh has the
// node layout, the rule for a closest hit and why its answer is the reference's), for the
// persistent kernel of walk.cuh.
//
// Against the walk of both kinds in one kernel: any-hit rays carry no order, no nearest
// hit and no second hit; what is left of a node is two words (its first child and hit
// inner slots, its inner slots) that pending siblings need no header read for; its hit
// leaves are tested before its children; the answer's outputs are read once more from the
// nearest triangle at the end instead of carried along.
//
// Box test. Per axis A = RN(RN(o - r) * inv), B = s * inv as in trace_wide.cuh, but a
// plane's byte q goes into the float 2^15 + q (0x4700qq00) and stays there: t = RN((2^15 +
// q) * B + C -+ m), with C = RN(A - 2^15 B) and m = 2^-18 |A| + 2^-6 |B|. Roundings lose at
// most 8u |A| and (2^-9 + 2^-9 + 2^-13) |B| with u = 2^-24 (C's and C -+ m's of a sum
// that is 2^15 |B| large; the reference's own and the plane's are below 1100u |B|), a
// quarter of m: near values come out no later and far values no earlier than the
// reference's. The margin is 1/64 of a step of the grid, and the conversion by which each
// byte was a float of its own is gone. Rays are trusted (quant_trusted) when 2^15 B stays
// finite: components from 2^-58, origins and coordinates within 2^60; others take the
// binary walk at once.
//
// Measured: the secondary rays of a 1080p frame (5.1M any-hit, 1.9M bounces, 100,608
// triangles) 1.79 -> 1.31 ms, the any-hit rays alone 1.1 -> 0.83; 1M closest-hit rays
// 0.63 -> 0.51, any-hit 0.42 -> 0.31 ms. Instruction issue (70 %) and the ALU (61 %: bytes
// to floats, minima and maxima) bind it; 17 to 21 lanes of 32 are at work.
#pragma once
#include "common.cuh"
#include "trace_any.cuh"
#include "trace_wide.cuh"

namespace timrt {

constexpr float kQuantMargin = 0.015625f;   // 2^-6

// Byte k of w0 and of w1 as the floats 2^15 + q (0x4700qq00), packed.
__device__ __forceinline__ uint64_t qbytes15(uint32_t w0, uint32_t w1, uint32_t k) {
    uint64_t r;
    const uint32_t lo = __byte_perm(w0, 0x47000000u, 0x7504u | k << 4), hi = __byte_perm(w1, 0x47000000u, 0x7504u | k << 4);
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}

// An axis' coefficient and its addends for near and far planes, each in both halves.
struct QuantAxis { uint64_t B, An, Af; };
__device__ __forceinline__ QuantAxis quant_axis(uint32_t o, uint32_t e, float org, float inv) {
    const float B = __uint_as_float(e << 23) * inv;
    const float A = (__uint_as_float(o) - org) * inv;
    const float C = __fmaf_rn(-32768.0f, B, A);
    const float m = __fmaf_rn(fabsf(A), kWiden, fabsf(B) * kQuantMargin);
    return {pack2f(B, B), pack2f(C - m, C - m), pack2f(C + m, C + m)};
}

// Whether the box test holds for the ray (see the header).
__device__ __forceinline__ bool quant_trusted(const Ray& r) {
    constexpr float dlo = 3.469446951953614e-18f, ohi = 1.152921504606847e18f;   // 2^-58, 2^60
    return fabsf(r.dx) >= dlo && fabsf(r.dy) >= dlo && fabsf(r.dz) >= dlo &&      // false for NaN too
           fabsf(r.ox) <= ohi && fabsf(r.oy) <= ohi && fabsf(r.oz) <= ohi;
}

// Prepares a ray; one that is not trusted is done at once, with st.leaf = 1.
template <bool ANY>
__device__ __forceinline__ void quant_init(TravState& st, uint32_t bottom) {
    st.ix = 1.0f / st.r.dx;
    st.iy = 1.0f / st.r.dy;
    st.iz = 1.0f / st.r.dz;
    if (!ANY) {
        st.t1 = __int_as_float(0x7F800000);
        st.near2 = false;
        st.first = 8u;
    }
    st.oct = (__float_as_uint(st.r.dx) >> 31) | (__float_as_uint(st.r.dy) >> 31) << 1 | (__float_as_uint(st.r.dz) >> 31) << 2;
    st.top = bottom;
    st.rec0 = st.rec1 = 0u;   // the siblings to visit next: first child << 8 | hit inner slots; all inner slots
    st.hit = false;
    const bool ok = quant_trusted(st.r);
    st.leaf = ok ? 0u : 1u;
    st.node = ok ? 0u : kAnyIdle;
}

// The next of the siblings in hand, or of the last ones put on the stack. Closest-hit rays
// take the node's nearest box first if it is an inner one (1.45 -> 1.38 ms for the frame's
// secondary rays), then the slots in the order of the ray's octant: children were placed
// by their direction from the node's centre.
template <int BLOCK, bool ANY>
__device__ __forceinline__ void quant_next(TravState& st, uint32_t bottom) {
    if (!(st.rec0 & 0xFFu)) {
        if (st.top == bottom) {
            st.node = kAnyIdle;
            return;
        }
        st.rec1 = stack_pop<BLOCK>(st.top);
        st.rec0 = stack_pop<BLOCK>(st.top);
        if (!ANY) st.first = 8u;
    }
    const uint32_t hits = st.rec0 & 0xFFu;
    uint32_t slot;
    if (ANY) {
        slot = (uint32_t)__ffs((int)hits) - 1u;
    } else if (st.first < 8u && (hits >> st.first & 1u)) {
        slot = st.first;
        st.first = 8u;
    } else {
        uint32_t h = hits;   // left with the slot whose slot ^ octant is the lowest
        const uint32_t oct = st.oct;
        if (oct & 4u) { if (h & 0xF0u) h &= 0xF0u; } else { if (h & 0x0Fu) h &= 0x0Fu; }
        if (oct & 2u) { if (h & 0xCCu) h &= 0xCCu; } else { if (h & 0x33u) h &= 0x33u; }
        if (oct & 1u) { if (h & 0xAAu) h &= 0xAAu; } else { if (h & 0x55u) h &= 0x55u; }
        slot = (uint32_t)__ffs((int)h) - 1u;
    }
    st.rec0 &= ~(1u << slot);
    st.node = (st.rec0 >> 8) + (uint32_t)__popc(st.rec1 & ((1u << slot) - 1u));
}

// One advance of one lane from the inner node st.node: its hit inner slots become the
// siblings in hand (those in hand before go onto the stack), its hit leaf slots the lane's
// leaf, bit 31 | node << 8 | slots.
template <int BLOCK, bool ANY>
__device__ __forceinline__ void quant_advance(TravState& st, const char* wnodes, uint32_t bottom) {
    const uint4* np = reinterpret_cast<const uint4*>(wnodes) + 5ull * st.node;
    const uint4 U0 = __ldg(np), U2 = __ldg(np + 2), U3 = __ldg(np + 3), U4 = __ldg(np + 4);
    const uint32_t child_base = __ldg(reinterpret_cast<const uint32_t*>(np) + 4);
    const QuantAxis X = quant_axis(U0.x, U0.w & 0xFFu, st.r.ox, st.ix);
    const QuantAxis Y = quant_axis(U0.y, (U0.w >> 8) & 0xFFu, st.r.oy, st.iy);
    const QuantAxis Z = quant_axis(U0.z, (U0.w >> 16) & 0xFFu, st.r.oz, st.iz);
    const bool negx = st.ix < 0.0f, negy = st.iy < 0.0f, negz = st.iz < 0.0f;
    const uint32_t nx0 = negx ? U3.z : U2.x, nx1 = negx ? U3.w : U2.y, fx0 = negx ? U2.x : U3.z, fx1 = negx ? U2.y : U3.w;
    const uint32_t ny0 = negy ? U4.x : U2.z, ny1 = negy ? U4.y : U2.w, fy0 = negy ? U2.z : U4.x, fy1 = negy ? U2.w : U4.y;
    const uint32_t nz0 = negz ? U4.z : U3.x, nz1 = negz ? U4.w : U3.y, fz0 = negz ? U3.x : U4.z, fz1 = negz ? U3.y : U4.w;
    const uint32_t imask = U0.w >> 24;
    uint32_t half[2] = {0u, 0u}, nearest = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t kk = 3; kk < 4u; --kk) {
        float a[2], b[2], c[2], d[2], e[2], f[2];
        unpack2f(fma2(qbytes15(nx0, nx1, kk), X.B, X.An), a[0], a[1]);
        unpack2f(fma2(qbytes15(fx0, fx1, kk), X.B, X.Af), d[0], d[1]);
        unpack2f(fma2(qbytes15(ny0, ny1, kk), Y.B, Y.An), b[0], b[1]);
        unpack2f(fma2(qbytes15(fy0, fy1, kk), Y.B, Y.Af), e[0], e[1]);
        unpack2f(fma2(qbytes15(nz0, nz1, kk), Z.B, Z.An), c[0], c[1]);
        unpack2f(fma2(qbytes15(fz0, fz1, kk), Z.B, Z.Af), f[0], f[1]);
        float tn[2], tf[2], gap[2];
#pragma unroll
        for (uint32_t h2 = 0; h2 < 2u; ++h2) {
            tn[h2] = max3f(fmaxf(a[h2], b[h2]), c[h2], 0.0f);
            tf[h2] = min3f(fminf(d[h2], e[h2]), f[h2], st.t);
        }
        unpack2f(sub2(pack2f(tn[0], tn[1]), pack2f(tf[0], tf[1])), gap[0], gap[1]);
#pragma unroll
        for (uint32_t h2 = 0; h2 < 2u; ++h2) {
            half[h2] = __funnelshift_l(__float_as_uint(gap[h2]), half[h2], 1u);   // entered where negative
            const uint32_t k = kk + 4u * h2;
            if (!ANY) nearest = min(nearest, gap[h2] < 0.0f  ? (__float_as_uint(tn[h2]) & ~7u) | k : 0xFFFFFFFFu);
        }
    }
    const uint32_t mask = half[0] | half[1] << 4;
    const uint32_t inner = mask & imask, leaves = mask & ~imask;
    if (inner) {
        if (st.rec0 & 0xFFu) {
            stack_push<BLOCK>(st.top, st.rec0, true);
            stack_push<BLOCK>(st.top, st.rec1, true);
        }
        st.rec0 = child_base << 8 | inner;
        st.rec1 = imask;
        if (!ANY) st.first = nearest & 7u;
    }
    if (leaves) st.node = 0x80000000u | st.node << 8 | leaves;
    else quant_next<BLOCK, ANY>(st, bottom);
}

// The triangles of the first slot of a leaf reference, and their number.
__device__ __forceinline__ uint32_t quant_leaf(const SceneView& s, uint32_t ref, uint32_t& first) {
    const uint32_t slot = (uint32_t)__ffs((int)(ref & 0xFFu)) - 1u;
    const uint4 U1 = __ldg(s.wnodes + 5ull * ((ref >> 8) & kQuantNodes) + 1);
    const uint64_t meta = (uint64_t)U1.w << 32 | U1.z, below = meta & ((1ull << (8u * slot)) - 1ull);
    first = U1.y + __dp4a((uint32_t)below, 0x01010101u, __dp4a((uint32_t)(below >> 32), 0x01010101u, 0u));
    return (uint32_t)(meta >> (8u * slot)) & 0xFFu;
}

// A hit below the closest-hit ray's bound st.t (see wide_leaf).
__device__ __forceinline__ void quant_hit(const float4* wtris, TravState& st, uint32_t tri, float t, bool dup_ok) {
    if (t < st.t1) {
        st.near2 = st.t1 - kOffsetRayCollision <= t;
        st.t1 = t;
        st.t = fminf(st.t, t + (kOffsetRayCollision + (t * 9.5367431640625e-07f + 9.313225746154785e-10f)));
        st.nid = tri;
        st.hit = true;
    } else if (!st.near2 && t - kOffsetRayCollision <= st.t1) {
        bool same = false;
        if (dup_ok && t == st.t1) {
            const float4 *a = wtris + 3ull * tri, *b = wtris + 3ull * st.nid;
            same = __float_as_uint(__ldg(a).w) == __float_as_uint(__ldg(b).w) &&
                   __float_as_uint(__ldg(a + 1).w) == __float_as_uint(__ldg(b + 1).w) &&
                   __float_as_uint(__ldg(a + 2).w) == __float_as_uint(__ldg(b + 2).w);
        }
        st.near2 = !same;
    }
}

// A leaf slot's triangles in their stored order on the ray's own lane (see wide_leaf).
template <bool ANY>
__device__ __forceinline__ bool quant_triangles(const float4* wtris, TravState& st, const Ray& r, uint32_t first, uint32_t cnt,
                                                bool dup_ok) {
    const float4* tp = wtris + 3ull * first;
    for (uint32_t i = 0; i < cnt; ++i, tp += 3) {
        const float4 A = __ldg(tp), B = __ldg(tp + 1), C = __ldg(tp + 2);
        float u, v;
        const float t = collide_triangle_e(r, A.x, A.y, A.z, B.x, B.y, B.z, C.x, C.y, C.z, st.t, u, v);
        if (t > 0.0f) {
            if (ANY) {
                st.nid = first + i;
                return true;
            }
            quant_hit(wtris, st, first + i, t, dup_ok);
        }
    }
    return false;
}

// The ray's answer where it stands (wide_finish; an any-hit ray as in any_finish), the
// binary walk's otherwise.
template <bool ANY>
__device__ __forceinline__ void quant_finish(const SceneView& s, TravState& st, bool want_bary, uint32_t* err) {
    bool same;
    const uint32_t tri = st.nid;
    if (!st.hit) {
        same = st.leaf == 0u;
        st.rec0 = st.rec1 = st.rec2 = 0u;
        st.u = st.v = 0.0f;
        st.nid = 0xFFFFFFFFu;
    } else {
        const uint4 lo = __ldg(s.wtri_leaf + 2ull * tri), hi = __ldg(s.wtri_leaf + 2ull * tri + 1u);
        same = false;
        if (hi.w == 0u) {
            const float lx = __uint_as_float(lo.x), ly = __uint_as_float(lo.y), lz = __uint_as_float(lo.z);
            const float hx = __uint_as_float(hi.x), hy = __uint_as_float(hi.y), hz = __uint_as_float(hi.z);
            constexpr float e = 4.76837158203125e-07f, a = 7.888609052210118e-31f;   // 2^-21, 2^-100
            const float ax = (lx - st.r.ox) * st.ix, bx = (hx - st.r.ox) * st.ix;
            const float ay = (ly - st.r.oy) * st.iy, by = (hy - st.r.oy) * st.iy;
            const float az = (lz - st.r.oz) * st.iz, bz = (hz - st.r.oz) * st.iz;
            const float sx = fminf(ax, bx), sy = fminf(ay, by), sz = fminf(az, bz);
            const float fx = fmaxf(ax, bx), fy = fmaxf(ay, by), fz = fmaxf(az, bz);
            const float up = fmaxf(0.0f, fmaxf(sx + fabsf(sx) * e, fmaxf(sy + fabsf(sy) * e, sz + fabsf(sz) * e))) + a;
            const float dn = fminf(fx - fabsf(fx) * e, fminf(fy - fabsf(fy) * e, fz - fabsf(fz) * e)) - a;
            if (ANY) {
                same = up < dn && up < st.t;
                if (!same) same = collide_box(st.r, lx, ly, lz, hx, hy, hz, st.t) >= 0.0f;
            } else {
                same = up <= st.t1 && up < dn;
                if (!same) {
                    const float d = collide_box(st.r, lx, ly, lz, hx, hy, hz, st.t0);
                    same = d >= 0.0f && d <= st.t1;
                }
            }
        }
        if (!ANY) {
            same = same && !st.near2;
            if (same) {
                const float4* tp = s.wtris + 3ull * tri;
                const float4 A = __ldg(tp), B = __ldg(tp + 1), C = __ldg(tp + 2);
                st.rec0 = __float_as_uint(A.w);
                st.rec1 = __float_as_uint(B.w);
                st.rec2 = __float_as_uint(C.w);
                st.nid = lo.w;
                st.u = st.v = 0.0f;
                if (want_bary)
                    collide_triangle_e(st.r, A.x, A.y, A.z, B.x, B.y, B.z, C.x, C.y, C.z, __int_as_float(0x7F800000), st.u, st.v);
                st.t = st.t1 - kOffsetRayCollision;
            }
        }
    }
    if (!same) {
        const BinaryResult b = binary_walk(s.nodes, s.leaf, s.pos, s.blas, s.num_nodes, s.leaf_words, st.r.ox, st.r.oy,
                                           st.r.oz, st.r.dx, st.r.dy, st.r.dz, ANY ? st.t : st.t0, ANY, err);
        if (!ANY) {
            st.rec0 = b.rec0; st.rec1 = b.rec1; st.rec2 = b.rec2; st.nid = b.nid;
            st.t = b.t; st.u = b.u; st.v = b.v;
        }
        st.hit = b.hit != 0u;
    }
}

}  // namespace timrt
