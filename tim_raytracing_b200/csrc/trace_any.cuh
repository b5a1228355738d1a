// trace_any.cuh -- any-hit rays on a 4-wide BVH with full-precision child boxes.
//
// An any-hit ray's answer does not depend on the order of its walk: its tmax is
// fixed, so the reference (traverseBvhFast, bvhTraversal_inline.glsl:83-151)
// reports a hit exactly when some triangle that CollideTriangle accepts lies in a
// leaf whose box and whose ancestors' boxes all pass CollideBox with that tmax.
// The walk here therefore uses a tree of its own over the reference's leaves
// (bvh_four.cu collapses the binary tree), with a box test that only has to accept
// every box the reference accepts, and checks at the end that the binary walk
// reaches the leaf of the hit it found.
//
// Node layout (224 B, built by bvh_four.cu):
//   per axis, 4 x float4: lo[4] hi[4] hi[4] lo[4], one word per slot
//   uint4   the slots' references: an inner node's index and the levels below it
//           (four_stack.h), or a leaf as bit 31 | triangles << 27 | first triangle (triangles 0: more than
//           15, read from the leaf's record); empty slots have inverted boxes
//   16 B    unused
// A ray reads its near and far planes of an axis, in this order, with one 32-byte
// load: from the first pair where its direction is positive, from the second where
// it is negative. That replaces the reference's min and max per axis (which run at
// half the rate of the multiply-adds on this GPU; the binary walk was bound by them),
// and one address per axis serves both planes. The odd multiple of 32 B puts the
// same axis of neighbouring nodes into different banks of the L1.
//
// Box test, and why it accepts every box the reference accepts. With inv within
// 2u of 1/d (u = 2^-24) and W = max(2^-20 (P + |o|), 2^-60), where P is the largest magnitude of any plane
// of the tree on that axis, a near plane is t = RN(p * inv + An), a far plane
// RN(p * inv + Af), An and Af being -o * inv less and plus m = W |inv|. Against the
// exact (p - o) / d the reciprocal, the addend's roundings and the final one lose
// at most 5u (P + |o|) |inv|, and the reference's own subtraction and division 2u
// of the same: m, 16u of it, is more than twice their sum, so near values come out
// no later and far values no earlier than the reference's. A zero component is
// replaced by +-2^-80: where the origin lies between the planes (the reference's
// slab is unbounded there) the near value is negative and the far one at least
// m / 2, which any_init requires to exceed every t at which a box can be entered;
// where it lies outside them the reference rejects the box anyway. Rays outside
// the stated ranges (any_init) take the binary walk.
//
// Why the answer is the reference's. No hit: the walk visits a superset of the
// reference's leaves, all with the same tmax and the same triangle test. A hit: the
// intersection E of the hit leaf's box and all its ancestors' boxes passes
// CollideBox with the ray's tmax; entry distances only fall and exits only grow
// from E to each of those boxes (IEEE subtraction and division are monotonic, and
// on an axis with a zero component an origin strictly inside E is strictly inside
// each of them), so the reference reaches the leaf too. A ray whose hit cannot be
// shown this way is traced again by the binary walk.
//
// Measured (1080p frame of the 100K-triangle scene, 5.1M any-hit rays; 6.6M of the
// 1279x719 frame with probe visibility): 1.07 -> 0.75 and 1.32 -> 0.94 ms against the
// binary walk, with half the node visits (10.7 against 20.3 a ray) and 30 % fewer
// instructions (0.69 ms for the former since; four_stack.h has scenes of overlapping
// boxes). The L1 binds it: 71 % of its data path's cycles, 61 % hits.
#pragma once
#include "common.cuh"
#include "four_stack.h"
#include "trace_plain.cuh"
#include "trace_wide.cuh"

namespace timrt {

constexpr float kFourZero = 8.271806125530277e-25f;      // 2^-80, stands in for a zero component
constexpr float kFourMargin = 9.5367431640625e-07f;      // 2^-20
constexpr float kFourFloor = 8.673617379884035e-19f;     // 2^-60
constexpr uint32_t kAnyIdle = 0xFFFFFFFFu;               // in place of a node: the ray's walk is over

// 1 / x to 1 ulp (MUFU.RCP), for x of ordinary magnitude.
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// Three-input max / min that return NaN when an operand is NaN.
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
    float r;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Prepares an any-hit ray. A ray that the box test's bounds do not cover is done at
// once, with st.leaf = 1: any_finish sends it to the binary walk.
__device__ __forceinline__ void any_init(const SceneView& s, TravState& st, uint32_t bottom) {
    constexpr float dlo = 8.673617379884035e-19f, dhi = 1.152921504606847e18f, ohi = 1.099511627776e12f;   // 2^+-60, 2^40
    const bool zx = st.r.dx == 0.0f, zy = st.r.dy == 0.0f, zz = st.r.dz == 0.0f;
    const float ux = zx ? copysignf(kFourZero, st.r.dx) : st.r.dx;
    const float uy = zy ? copysignf(kFourZero, st.r.dy) : st.r.dy;
    const float uz = zz ? copysignf(kFourZero, st.r.dz) : st.r.dz;
    st.ix = rcp_fast(ux);
    st.iy = rcp_fast(uy);
    st.iz = rcp_fast(uz);
    const float rx = s.bound4[0] + fabsf(st.r.ox), ry = s.bound4[1] + fabsf(st.r.oy), rz = s.bound4[2] + fabsf(st.r.oz);
    const float mx = fmaxf(rx * kFourMargin, kFourFloor) * fabsf(st.ix);
    const float my = fmaxf(ry * kFourMargin, kFourFloor) * fabsf(st.iy);
    const float mz = fmaxf(rz * kFourMargin, kFourFloor) * fabsf(st.iz);
    const float ax = st.r.ox * st.ix, ay = st.r.oy * st.iy, az = st.r.oz * st.iz;
    st.anx = -ax - mx; st.any_ = -ay - my; st.anz = -az - mz;
    st.afx = mx - ax; st.afy = my - ay; st.afz = mz - az;
    const char* base = reinterpret_cast<const char*>(s.nodes4);
    st.px = base + (st.ix < 0.0f ? 32u : 0u);
    st.py = base + (st.iy < 0.0f ? 96u : 64u);
    st.pz = base + (st.iz < 0.0f ? 160u : 128u);
    st.refs = base + 192u;
    const float fx = fabsf(ux), fy = fabsf(uy), fz = fabsf(uz);
    bool ok = max3_nan(fx, fy, fz) <= dhi && max3_nan(fabsf(st.r.ox), fabsf(st.r.oy), fabsf(st.r.oz)) <= ohi && st.t == st.t;
    if (!(min3_nan(fx, fy, fz) >= dlo)) {   // a zero component, or one too small
        // no box is entered later than the ray leaves the tree's bounds on any axis it moves along
        ok = ok && (zx || fx >= dlo) && (zy || fy >= dlo) && (zz || fz >= dlo);
        float tb = st.t;
        if (!zx) tb = fminf(tb, 1.01f * rx * fabsf(st.ix));
        if (!zy) tb = fminf(tb, 1.01f * ry * fabsf(st.iy));
        if (!zz) tb = fminf(tb, 1.01f * rz * fabsf(st.iz));
        tb *= 2.0f;
        ok = ok && (!zx || mx >= tb) && (!zy || my >= tb) && (!zz || mz >= tb);
    }
    st.top = bottom;
    st.hit = false;
    st.leaf = ok ? 0u : 1u;
    st.node = ok ? (s.depth4 - 1u) << kFourBelowShift : kAnyIdle;
}

// Eight floats at a 32-byte boundary.
__device__ __forceinline__ void load8(const char* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// The walks' stacks, by shared-memory address: word k of a thread lies 4 * BLOCK bytes
// above word k - 1. A push writes above the top and moves it when `keep`.
template <int BLOCK>
__device__ __forceinline__ void stack_push(uint32_t& top, uint32_t v, bool keep) {
    asm volatile("st.shared.b32 [%0 + %2], %1;" ::"r"(top), "r"(v), "n"(4 * BLOCK) : "memory");
    if (keep) top += 4u * BLOCK;
}
template <int BLOCK>
__device__ __forceinline__ uint32_t stack_pop(uint32_t& top) {
    uint32_t v;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(top) : "memory");
    top -= 4u * BLOCK;
    return v;
}

// What only leaves and ends of walks need of a ray lies in shared memory while it is
// under way, word k of thread t at [k * BLOCK + t]: held in registers it made the
// node visits spill.
template <int BLOCK>
__device__ __forceinline__ void put3(uint32_t* p, float x, float y, float z) {
    p[0] = __float_as_uint(x);
    p[BLOCK] = __float_as_uint(y);
    p[2 * BLOCK] = __float_as_uint(z);
}
template <int BLOCK>
__device__ __forceinline__ void get3(const uint32_t* p, float& x, float& y, float& z) {
    x = __uint_as_float(p[0]);
    y = __uint_as_float(p[BLOCK]);
    z = __uint_as_float(p[2 * BLOCK]);
}

// The references of node 0.
__device__ __forceinline__ const char* four_refs(const SceneView& s) {
    return reinterpret_cast<const char*>(s.nodes4) + 192u;
}

// A slot's box test (see the header).
struct AnyBoxRay { float ix, iy, iz, anx, any_, anz, afx, afy, afz, t; };
template <class R>
__device__ __forceinline__ bool any_enters(const R& r, float nx, float fx, float ny, float fy, float nz, float fz) {
    const float tn = max3f(fmaxf(__fmaf_rn(nx, r.ix, r.anx), __fmaf_rn(ny, r.iy, r.any_)), __fmaf_rn(nz, r.iz, r.anz), 0.0f);
    const float tf = min3f(fminf(__fmaf_rn(fx, r.ix, r.afx), __fmaf_rn(fy, r.iy, r.afy)), __fmaf_rn(fz, r.iz, r.afz), r.t);
    return tn < tf;
}

// The entered slots of a node: any_advance's box tests where the slots don't fit on the
// stack.
static __device__ __forceinline__ uint32_t any_slots(AnyBoxRay r, const char* px, const char* py, const char* pz) {
    float4 nx, fx, ny, fy, nz, fz;
    load8(px, nx, fx);
    load8(py, ny, fy);
    load8(pz, nz, fz);
    return (any_enters(r, nx.x, fx.x, ny.x, fy.x, nz.x, fz.x) ? 1u : 0u) | (any_enters(r, nx.y, fx.y, ny.y, fy.y, nz.y, fz.y) ? 2u : 0u) |
           (any_enters(r, nx.z, fx.z, ny.z, fy.z, nz.z, fz.z) ? 4u : 0u) | (any_enters(r, nx.w, fx.w, ny.w, fy.w, nz.w, fz.w) ? 8u : 0u);
}

// any_advance from a node whose slots don't fit on the stack, or that waits (four_stack.h).
template <int BLOCK>
__device__ __forceinline__ void any_advance_tight(TravState& st, const char* refs_base) {
    if (!(st.node & kFourWaiting)) {
        const uint64_t off = (uint64_t)(st.node & kFourIndexMask) * kFourBytes;
        const uint32_t slots = any_slots(AnyBoxRay{st.ix, st.iy, st.iz, st.anx, st.any_, st.anz, st.afx, st.afy, st.afz, st.t},
                                         st.px + off, st.py + off, st.pz + off);
        st.node = slots ? four_waiting(st.node, slots) : stack_pop<BLOCK>(st.top);
        return;
    }
    const uint32_t slot = 31u - (uint32_t)__clz((int)(st.node & 15u)), rest = st.node & ~(1u << slot);   // the last of them
    stack_push<BLOCK>(st.top, rest, (rest & 15u) != 0u);
    st.node = __ldg(reinterpret_cast<const uint32_t*>(refs_base + (uint64_t)((st.node >> 4) & kFourIndexMask) * kFourBytes) + slot);
}

// One advance of one lane from the inner node st.node: its slots whose boxes are
// entered go onto the stack, smallest box first, and the last one is taken. (The
// entered box nearest first instead: 6 % fewer visits, but 20 more instructions each.)
template <int BLOCK>
__device__ __forceinline__ void any_advance(TravState& st, const char* refs_base, uint32_t near, uint32_t bottom, int sdepth) {
    if (st.top >= near && !four_fits(st.top, st.node, bottom, sdepth, 4u * BLOCK)) {
        any_advance_tight<BLOCK>(st, refs_base);
        return;
    }
    const uint64_t off = (uint64_t)(st.node & kFourIndexMask) * kFourBytes;
    float4 nx, fx, ny, fy, nz, fz;
    load8(st.px + off, nx, fx);
    load8(st.py + off, ny, fy);
    load8(st.pz + off, nz, fz);
    const uint4 ref = __ldg(reinterpret_cast<const uint4*>(refs_base + off));
    stack_push<BLOCK>(st.top, ref.x, any_enters(st, nx.x, fx.x, ny.x, fy.x, nz.x, fz.x));
    stack_push<BLOCK>(st.top, ref.y, any_enters(st, nx.y, fx.y, ny.y, fy.y, nz.y, fz.y));
    stack_push<BLOCK>(st.top, ref.z, any_enters(st, nx.z, fx.z, ny.z, fy.z, nz.z, fz.z));
    stack_push<BLOCK>(st.top, ref.w, any_enters(st, nx.w, fx.w, ny.w, fy.w, nz.w, fz.w));
    st.node = stack_pop<BLOCK>(st.top);
}

// The triangles of a leaf reference, and their number.
__device__ __forceinline__ uint32_t leaf_ref(const SceneView& s, uint32_t ref, uint32_t& first) {
    first = ref & kFourFirstMask;
    uint32_t cnt = (ref >> kFourCountShift) & 15u;
    if (cnt == 0u && first != kFourFirstMask)   // not the closest-hit records' empty leaf
        cnt = __ldg(reinterpret_cast<const uint32_t*>(s.leaf4 + 2u * __ldg(s.tri_leaf4 + first) + 1u) + 3) >> 2;
    return cnt;
}

// A leaf's triangles in their stored order on the ray's own lane: an any-hit ray's first
// hit (bvh_collide_fast, bvhCollision.glsl:241-284; returns true), or every hit of a
// closest-hit ray below t, which it shrinks to 1e-5 under the hit (bvh_collide,
// bvhCollision.glsl:177-239).
template <bool ANY>
__device__ __forceinline__ bool leaf_triangles(const float4* ptris, TravState& st, const Ray& r, uint32_t first, uint32_t cnt) {
    const float4* tp = ptris + 3ull * first;
    for (uint32_t i = 0; i < cnt; ++i, tp += 3) {
        const float4 A = __ldg(tp), B = __ldg(tp + 1), C = __ldg(tp + 2);
        float u, v;
        const float t = collide_triangle_e(r, A.x, A.y, A.z, B.x, B.y, B.z, C.x, C.y, C.z, st.t, u, v);
        if (t > 0.0f) {
            st.nid = first + i;
            if (ANY) return true;
            st.t = t - kOffsetRayCollision;
            st.hit = true;
        }
    }
    return false;
}

// Whether the ray's answer stands (see the header): no hit, or a hit in a leaf that
// the binary walk reaches.
__device__ __forceinline__ bool any_finish(const SceneView& s, const TravState& st) {
    if (!st.hit) return st.leaf == 0u;
    const uint32_t l = __ldg(s.tri_leaf4 + st.nid);
    const uint4 lo = __ldg(s.leaf4 + 2u * l), hi = __ldg(s.leaf4 + 2u * l + 1u);
    if (hi.w & 3u) return false;   // the boxes on its path do not overlap
    const float lx = __uint_as_float(lo.x), ly = __uint_as_float(lo.y), lz = __uint_as_float(lo.z);
    const float hx = __uint_as_float(hi.x), hy = __uint_as_float(hi.y), hz = __uint_as_float(hi.z);
    if ((st.r.dx == 0.0f && !(lx < st.r.ox && st.r.ox < hx)) || (st.r.dy == 0.0f && !(ly < st.r.oy && st.r.oy < hy)) ||
        (st.r.dz == 0.0f && !(lz < st.r.oz && st.r.oz < hz)))
        return false;
    // By multiplication first, entries moved up and exits down by 2^-21 of their
    // magnitude (wide_finish has the argument); the reference's divisions otherwise.
    constexpr float e = 4.76837158203125e-07f, a = 7.888609052210118e-31f;   // 2^-21, 2^-100
    const float ax = (lx - st.r.ox) * st.ix, bx = (hx - st.r.ox) * st.ix;
    const float ay = (ly - st.r.oy) * st.iy, by = (hy - st.r.oy) * st.iy;
    const float az = (lz - st.r.oz) * st.iz, bz = (hz - st.r.oz) * st.iz;
    const float sx = fminf(ax, bx), sy = fminf(ay, by), sz = fminf(az, bz);
    const float fx = fmaxf(ax, bx), fy = fmaxf(ay, by), fz = fmaxf(az, bz);
    const float up = fmaxf(0.0f, fmaxf(sx + fabsf(sx) * e, fmaxf(sy + fabsf(sy) * e, sz + fabsf(sz) * e))) + a;
    const float dn = fminf(fx - fabsf(fx) * e, fminf(fy - fabsf(fy) * e, fz - fabsf(fz) * e)) - a;
    if (up < dn && up < st.t) return true;
    return collide_box(st.r, lx, ly, lz, hx, hy, hz, st.t) >= 0.0f;
}

// any_finish, and the binary walk when it fails: afterwards st.hit is the reference's answer.
__device__ __forceinline__ void any_finish_or_walk(const SceneView& s, TravState& st, uint32_t* err) {
    if (any_finish(s, st)) return;
    const BinaryResult b = binary_walk(s.nodes, s.leaf, s.pos, s.blas, s.num_nodes, s.leaf_words, st.r.ox, st.r.oy,
                                       st.r.oz, st.r.dx, st.r.dy, st.r.dz, st.t, true, err);
    st.hit = b.hit != 0u;
}

}  // namespace timrt
