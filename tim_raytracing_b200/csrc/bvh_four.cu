// bvh_four.cu -- the trees the binary form's rays walk, built on the GPU from an uploaded
// scene's binary tree: the leaf triangles by node, the 4-wide tree of the any-hit rays
// (trace_any.cuh) and the child-pair records of the closest-hit rays (trace_pair.cuh).
//
// Every 4-wide slot is one binary subtree, so a leaf of the 4-wide tree is a leaf of
// the reference's with its triangles in their order. Which subtrees become a node's
// slots is the cut of least surface-area cost: cost[x][k], the least summed area of
// inner nodes when the subtree of x is covered by at most k slots, is filled
// bottom-up (the second child to arrive merges, after a fence), then the nodes are
// numbered level by level from the root and written. The collapse of the 8-wide
// form does the same on the host; here it adds four short kernels and one launch a
// level to an upload (1M triangles: under a millisecond of device time) and no host
// work.
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include "common.cuh"
#include "context.h"
#include "four_stack.h"
#include "kernels.h"

namespace timrt {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kMaxLevels = kStackSize + 1;

// Counters of one build.
struct Ctl {
    uint32_t total;                    // 4-wide nodes numbered so far
    uint32_t leaves;                   // leaf slots
    uint32_t bad;                      // a shared child, a non-finite plane, or more nodes than the tree has
    uint32_t ticket;
    uint32_t level[kMaxLevels + 2];    // first node of each level
    uint32_t bound[3];                 // bits of the largest magnitude of any plane, per axis
};

struct In {
    const float4* nodes;
    const uint4* pleaf;      // per node: (first triangle, leaf header, ...)
    uint32_t num_nodes;
};

struct Box { float lo[3], hi[3]; };

// A subtree on its way into a slot: node id | leaf bit, slots it may take, its stored
// box and the intersection E of that box and its ancestors'.
struct Sub {
    uint32_t id;
    int k;
    Box box, e;
};

__device__ __forceinline__ uint32_t children_of(const In& in, uint32_t x) {
    return reinterpret_cast<const uint4*>(in.nodes + 4u * x)->z;
}

__device__ __forceinline__ void child_boxes(const In& in, uint32_t x, Box& l, Box& r) {
    const float4 a = in.nodes[4u * x + 1u], b = in.nodes[4u * x + 2u], c = in.nodes[4u * x + 3u];
    const float la[6] = {a.x, a.y, c.x, a.z, a.w, c.y}, ra[6] = {b.x, b.y, c.z, b.z, b.w, c.w};
    for (int d = 0; d < 3; ++d) {   // the slab test orders each axis itself
        l.lo[d] = fminf(la[d], la[3 + d]); l.hi[d] = fmaxf(la[d], la[3 + d]);
        r.lo[d] = fminf(ra[d], ra[3 + d]); r.hi[d] = fmaxf(ra[d], ra[3 + d]);
    }
}

__device__ __forceinline__ uint32_t left_id(uint32_t packed) {
    return (packed & kNidMask) | (packed & kNidLeftLeafBit ? kNidLeafBit : 0u);
}
__device__ __forceinline__ uint32_t right_id(uint32_t packed) {
    return ((packed & kNidMask) + 1u) | (packed & kNidRightLeafBit ? kNidLeafBit : 0u);
}

__device__ __forceinline__ float area_of(const Box& b) {
    const float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
    return x * y + y * z + z * x;
}

// Least cost of covering a subtree with at most k = 0..4 slots. Leaves cost nothing
// (every cut of the tree holds all of them); a subtree without triangles takes no slot.
struct Cover { float f[5]; };

__device__ __forceinline__ Cover cover_of(const In& in, const float4* cost, uint32_t id) {
    Cover c;
    const uint32_t x = id & kNidMask;
    if (id & kNidLeafBit) {
        const bool empty = (in.pleaf[x].y & ((1u << kTriBits) - 1u)) == 0u;
        c.f[0] = empty ? 0.0f : INFINITY;
        c.f[1] = c.f[2] = c.f[3] = c.f[4] = 0.0f;
        return c;
    }
    const float4 v = __ldcg(cost + x);
    const bool empty = v.x < 0.0f;
    c.f[0] = empty ? 0.0f : INFINITY;
    c.f[1] = empty ? 0.0f : v.x;
    c.f[2] = empty ? 0.0f : v.y;
    c.f[3] = empty ? 0.0f : v.z;
    c.f[4] = empty ? 0.0f : v.w;
    return c;
}

// Best division of k slots between two subtrees: the cost, and the left one's share.
__device__ __forceinline__ float divide(const Cover& l, const Cover& r, int k, int& share) {
    float best = INFINITY;
    share = 0;
    for (int j = 0; j <= k; ++j) {
        const float v = l.f[j] + r.f[k - j];
        if (v < best) { best = v; share = j; }
    }
    return best;
}

__global__ void k_four_parents(In in, uint32_t* parent, Ctl* ctl) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    float m[3] = {0.f, 0.f, 0.f};
    bool bad = false;
    if (i < in.num_nodes) {
        const uint32_t c = children_of(in, i) & kNidMask;
        if (c != kNidMask) {
            bad = atomicCAS(parent + c, kNone, i) != kNone;
            bad |= atomicCAS(parent + c + 1u, kNone, i) != kNone;
            Box b[2];
            child_boxes(in, i, b[0], b[1]);
            for (int s = 0; s < 2; ++s)
                for (int d = 0; d < 3; ++d) {
                    // fminf / fmaxf drop a single NaN: look at the raw planes too
                    m[d] = fmaxf(m[d], fmaxf(fabsf(b[s].lo[d]), fabsf(b[s].hi[d])));
                }
            for (int w = 1; w < 4; ++w) {
                const float4 v = in.nodes[4u * i + w];
                bad |= !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w));
            }
        }
    }
    for (int d = 0; d < 3; ++d) {
        const uint32_t v = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(m[d]));
        if ((threadIdx.x & 31u) == 0u && v) atomicMax(ctl->bound + d, v);
    }
    if (bad) atomicOr(&ctl->bad, 1u);
}

// From each leaf up: the second arrival at a node fills its costs and goes on.
__global__ void k_four_cost(In in, const uint32_t* parent, uint32_t* arrivals, float4* cost, const Ctl* ctl) {
    if (ctl->bad) return;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= in.num_nodes) return;
    uint32_t x = i;
    uint32_t p = parent[x];
    if (p == kNone) return;
    uint32_t packed = children_of(in, p);
    if (!((x == (packed & kNidMask) ? left_id(packed) : right_id(packed)) & kNidLeafBit)) return;   // not a leaf
    for (;;) {
        __threadfence();
        if (atomicAdd(arrivals + p, 1u) == 0u) return;
        __threadfence();
        const Cover l = cover_of(in, cost, left_id(packed)), r = cover_of(in, cost, right_id(packed));
        const uint32_t pp = parent[p];
        uint32_t up = 0;
        float area = 0.0f;
        if (pp != kNone) {
            up = children_of(in, pp);
            Box a, b;
            child_boxes(in, pp, a, b);
            area = area_of(p == (up & kNidMask) ? a : b);
        }
        int j;
        const float single = area + divide(l, r, 4, j);
        float4 v = make_float4(-1.0f, 0.0f, 0.0f, 0.0f);   // no triangle below
        if (!(l.f[0] == 0.0f && r.f[0] == 0.0f))
            v = make_float4(fminf(single, divide(l, r, 1, j)), fminf(single, divide(l, r, 2, j)),
                            fminf(single, divide(l, r, 3, j)), fminf(single, divide(l, r, 4, j)));
        __stcg(cost + p, v);
        if (pp == kNone) return;
        if ((p == (up & kNidMask) ? left_id(up) : right_id(up)) & kNidLeafBit) return;   // used as a leaf above
        p = pp;
        packed = up;
    }
}

// The slots of the 4-wide node of binary node x (at most 4; leaves without triangles
// take none), by increasing area: the walk takes the last slot it entered first, and the largest is the likeliest occluder.
__device__ int expand(const In& in, const float4* cost, uint32_t x, const Box& e, Sub out[4]) {
    Sub st[4];   // the shares of the subtrees on it never sum to more than four
    int sp = 0, n = 0;
    auto push = [&](uint32_t node, int k, const Box& pe) {
        const uint32_t packed = children_of(in, node);
        Sub a, b;
        a.id = left_id(packed);
        b.id = right_id(packed);
        child_boxes(in, node, a.box, b.box);
        int j;
        divide(cover_of(in, cost, a.id), cover_of(in, cost, b.id), k, j);
        a.k = j;
        b.k = k - j;
        for (Sub* c : {&a, &b})
            for (int d = 0; d < 3; ++d) {
                c->e.lo[d] = fmaxf(pe.lo[d], c->box.lo[d]);
                c->e.hi[d] = fminf(pe.hi[d], c->box.hi[d]);
            }
        if (b.k) st[sp++] = b;   // a subtree without triangles takes no slot
        if (a.k) st[sp++] = a;
    };
    push(x, 4, e);
    while (sp > 0) {
        const Sub s = st[--sp];
        if (!(s.id & kNidLeafBit)) {
            const uint32_t packed = children_of(in, s.id);
            const Cover l = cover_of(in, cost, left_id(packed)), r = cover_of(in, cost, right_id(packed));
            if (l.f[0] == 0.0f && r.f[0] == 0.0f) continue;
            int j;
            if (divide(l, r, s.k, j) < area_of(s.box) + divide(l, r, 4, j)) {
                push(s.id, s.k, s.e);
                continue;
            }
        } else if ((in.pleaf[s.id & kNidMask].y & ((1u << kTriBits) - 1u)) == 0u) {
            continue;
        }
        int q = n++;
        for (; q > 0 && area_of(out[q - 1].box) > area_of(s.box); --q) out[q] = out[q - 1];
        out[q] = s;
    }
    return n;
}

// Node w of a level: its inner slots become nodes of the next one.
__device__ void four_node(const In& in, const float4* cost, uint32_t* item, Box* item_e, uint2* base, uint32_t cap, uint32_t w,
                          Ctl* ctl) {
    Sub s[4];
    const int n = expand(in, cost, item[w], item_e[w], s);
    uint32_t inner = 0;
    for (int k = 0; k < n; ++k) inner += s[k].id & kNidLeafBit ? 0u : 1u;
    const uint32_t first = inner ? atomicAdd(&ctl->total, inner) : 0u;
    const uint32_t leaf = inner < (uint32_t)n ? atomicAdd(&ctl->leaves, (uint32_t)n - inner) : 0u;
    base[w] = make_uint2(first, leaf);
    if (first + inner > cap) {
        atomicOr(&ctl->bad, 2u);
        return;
    }
    uint32_t q = first;
    for (int k = 0; k < n; ++k)
        if (!(s[k].id & kNidLeafBit)) {
            item[q] = s[k].id;
            item_e[q] = s[k].e;
            ++q;
        }
}

__global__ void __launch_bounds__(128) k_four_level(In in, const float4* cost, uint32_t* item, Box* item_e, uint2* base,
                                                    uint32_t cap, uint32_t lv, Ctl* ctl) {
    if (!ctl->bad) {
        const uint32_t end = ctl->level[lv + 1u];
        for (uint32_t w = ctl->level[lv] + blockIdx.x * blockDim.x + threadIdx.x; w < end; w += gridDim.x * blockDim.x)
            four_node(in, cost, item, item_e, base, cap, w, ctl);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1u) {
            ctl->ticket = 0u;
            ctl->level[lv + 2u] = *reinterpret_cast<volatile uint32_t*>(&ctl->total);
        }
    }
}

// All levels of a small tree by one block, instead of a launch per level of the binary tree,
// of which half are empty: the upload of 1,000 triangles 0.28 -> 0.25 ms, its second in a
// context 0.25 -> 0.21.
constexpr uint32_t kSmallTree = 2048u;   // inner binary nodes
__global__ void __launch_bounds__(256) k_four_small(In in, const float4* cost, uint32_t* item, Box* item_e, uint2* base,
                                                    uint32_t cap, uint32_t depth, Ctl* ctl) {
    uint32_t begin = 0u, end = 1u;
    for (uint32_t lv = 0; lv < depth && begin < end; ++lv) {
        if (!*reinterpret_cast<volatile uint32_t*>(&ctl->bad))
            for (uint32_t w = begin + threadIdx.x; w < end; w += blockDim.x) four_node(in, cost, item, item_e, base, cap, w, ctl);
        __syncthreads();
        begin = end;
        end = *reinterpret_cast<volatile uint32_t*>(&ctl->total);
        if (threadIdx.x == 0) ctl->level[lv + 2u] = end;
        __syncthreads();
    }
}

// The first node of each level.
struct Levels { uint32_t count, first[kMaxLevels]; };

__global__ void __launch_bounds__(128) k_four_fill(In in, const float4* cost, const uint32_t* item, const Box* item_e,
                                                   const uint2* base, uint32_t total, Levels levels, float4* nodes4,
                                                   uint4* leaf4, uint32_t* tri_leaf4) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= total) return;
    uint32_t below = 0;   // the levels after w's
    for (uint32_t lv = 1; lv < levels.count; ++lv) below += w < levels.first[lv] ? 1u : 0u;
    Sub s[4];
    const int n = expand(in, cost, item[w], item_e[w], s);
    uint2 b = base[w];
    float lo[3][4], hi[3][4];
    uint32_t ref[4];
    for (int k = 0; k < 4; ++k) {
        for (int d = 0; d < 3; ++d) {   // an empty slot's box is inverted
            lo[d][k] = k < n ? s[k].box.lo[d] : 1e30f;
            hi[d][k] = k < n ? s[k].box.hi[d] : -1e30f;
        }
        ref[k] = 0u;
        if (k >= n) continue;
        if (!(s[k].id & kNidLeafBit)) {
            ref[k] = (below - 1u) << kFourBelowShift | b.x++;   // an inner slot's node is of the next level
            continue;
        }
        const uint32_t nid = s[k].id & kNidMask;
        const uint4 li = in.pleaf[nid];
        const uint32_t nt = li.y & ((1u << kTriBits) - 1u);
        ref[k] = kNidLeafBit | (nt < 16u ? nt << kFourCountShift : 0u) | li.x;
        const Box& e = s[k].e;
        const bool empty = e.lo[0] > e.hi[0] || e.lo[1] > e.hi[1] || e.lo[2] > e.hi[2];
        leaf4[2u * b.y] = make_uint4(__float_as_uint(e.lo[0]), __float_as_uint(e.lo[1]), __float_as_uint(e.lo[2]), nid);
        leaf4[2u * b.y + 1u] = make_uint4(__float_as_uint(e.hi[0]), __float_as_uint(e.hi[1]), __float_as_uint(e.hi[2]),
                                          (empty ? 2u : 0u) | nt << 2);
        for (uint32_t t = 0; t < nt; ++t) tri_leaf4[li.x + t] = b.y;
        ++b.y;
    }
    float4* o = nodes4 + (kFourBytes / 16u) * (uint64_t)w;
    for (uint32_t d = 0; d < 3u; ++d) {
        o[4u * d] = o[4u * d + 3u] = make_float4(lo[d][0], lo[d][1], lo[d][2], lo[d][3]);
        o[4u * d + 1u] = o[4u * d + 2u] = make_float4(hi[d][0], hi[d][1], hi[d][2], hi[d][3]);
    }
    reinterpret_cast<uint4*>(o)[12] = make_uint4(ref[0], ref[1], ref[2], ref[3]);
    o[13] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The record of each inner node's children (trace_pair.cuh), at half the left one's id.
__global__ void k_pairs(In in, float4* pairs) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= in.num_nodes) return;
    const uint32_t packed = children_of(in, i), left = packed & kNidMask;
    if (left == kNidMask) return;
    Box b[2];
    child_boxes(in, i, b[0], b[1]);
    uint32_t ref[2];
    for (int k = 0; k < 2; ++k) {
        const uint32_t id = k ? right_id(packed) : left_id(packed), x = id & kNidMask;
        if (id & kNidLeafBit) {
            const uint4 li = in.pleaf[x];
            const uint32_t nt = li.y & ((1u << kTriBits) - 1u);
            ref[k] = nt == 0u ? kNidLeafBit | kFourFirstMask : kNidLeafBit | (nt < 16u ? nt << kFourCountShift : 0u) | li.x;
        } else {
            ref[k] = (children_of(in, x) & kNidMask) >> 1;   // validated: an inner node has children
        }
    }
    float4* o = pairs + (kPairBytes / 16u) * (uint64_t)(left >> 1);
    for (uint32_t d = 0; d < 3u; ++d) {
        o[2u * d] = make_float4(b[0].lo[d], b[1].lo[d], b[0].hi[d], b[1].hi[d]);
        o[2u * d + 1u] = make_float4(b[0].hi[d], b[1].hi[d], b[0].lo[d], b[1].lo[d]);
    }
    o[6] = make_float4(__uint_as_float(ref[0]), __uint_as_float(ref[1]), 0.f, 0.f);
}

// Per node (first triangle, leaf header, leaf-data offset, 0); a node without leaf data
// (offset 0xFFFFFFFF) gets header 0, as the kernels read it. Per leaf-data triangle
// record, in its leaf's order: (p0, vertexOffset) (p1 - p0, index01) (p2 - p0,
// index2_matId), the edges being the same rounded differences CollideTriangle forms
// (collision.glsl:60-61). A block takes the places of its nodes' triangles together
// (blocks in any order: nothing depends on it). Runs after validate_bvh, so every offset
// and vertex index is in range. The host loop this replaces and the copy of its result
// were half of a 1M-triangle scene's upload.
__global__ void __launch_bounds__(256) k_leaf_tris(SceneView s, uint32_t n, uint4* info, float4* tris) {
    __shared__ uint32_t warp_sum[8], block_base;
    const uint32_t i = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t off = 0xFFFFFFFFu, hdr = 0u;
    if (i < n) {
        off = reinterpret_cast<const uint4*>(s.nodes + 4u * i)->w;
        hdr = off == 0xFFFFFFFFu ? 0u : s.leaf[off];
    }
    const uint32_t nt = hdr & ((1u << kTriBits) - 1u);
    uint32_t sum = nt;
    for (uint32_t k = 1; k < 32u; k <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, sum, k);
        if (lane >= k) sum += v;
    }
    if (lane == 31u) warp_sum[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0u) {
        uint32_t t = 0;
        for (uint32_t k = 0; k < 8u; ++k) {
            const uint32_t v = warp_sum[k];
            warp_sum[k] = t;
            t += v;
        }
        block_base = t ? atomicAdd(&info[0].w, t) : 0u;
    }
    __syncthreads();
    if (i >= n) return;
    const uint32_t first = block_base + warp_sum[warp] + sum - nt;
    info[i].x = first;
    info[i].y = hdr;
    info[i].z = off;
    if (i) info[i].w = 0u;
    for (uint32_t t = 0; t < nt; ++t) {
        const uint32_t* r = s.leaf + 1u + off + 3u * t;
        const uint32_t r0 = r[0], r1 = r[1], r2 = r[2];
        const float* P0 = s.pos + 3ull * (r0 + (r1 & 0xFFFFu));
        const float* P1 = s.pos + 3ull * (r0 + (r1 >> 16));
        const float* P2 = s.pos + 3ull * (r0 + (r2 & 0xFFFFu));
        float4* o = tris + 3ull * (first + t);
        o[0] = make_float4(P0[0], P0[1], P0[2], __uint_as_float(r0));
        o[1] = make_float4(P1[0] - P0[0], P1[1] - P0[1], P1[2] - P0[2], __uint_as_float(r1));
        o[2] = make_float4(P2[0] - P0[0], P2[1] - P0[1], P2[2] - P0[2], __uint_as_float(r2));
    }
}

}  // namespace

cudaError_t build_leaf_tris(const Scene* s, cudaStream_t stream) {
    const uint32_t n = s->pc.numNodes;
    uint4* info = static_cast<uint4*>(s->pleaf.ptr);
    cudaMemsetAsync(info, 0, 16, stream);   // node 0's unused word counts the triangles handed out
    k_leaf_tris<<<(n + 255u) / 256u, 256, 0, stream>>>(s->view, n, info, static_cast<float4*>(s->ptris.ptr));
    return cudaGetLastError();
}

int build_four(tim_rt_ctx* c, Scene* s, uint64_t num_tris, uint32_t root_left) {
    const uint32_t n = s->pc.numNodes;
    // With a memory budget the scene keeps to the arrays it always had, so that what
    // was admitted stays admitted; BLAS boxes are tested by the binary walk only.
    if (c->budget || s->pc.numBlas || n < 2u || num_tris == 0u || num_tris >= kFourFirstMask) return TIM_RT_OK;
    auto up = [](uint64_t x) { return (x + 255ull) & ~255ull; };
    const uint32_t cap = n / 2u + 1u;   // inner nodes
    const uint64_t o_par = up(sizeof(Ctl)), o_arr = o_par + up(4ull * n), o_cost = o_arr + up(4ull * n),
                   o_item = o_cost + up(16ull * n), o_e = o_item + up(4ull * cap), o_base = o_e + up(sizeof(Box) * cap),
                   bytes = o_base + up(8ull * cap);
    // No room for the trees is no error: the plain walk stays.
    const std::string last_error = tim_rt_last_error();
    auto alloc = [&](DevBuf& b, uint64_t size) {
        if (dev_alloc(c, b, size) == TIM_RT_OK) return true;
        set_error(last_error);
        return false;
    };
    if (c->bld.bytes < bytes) {   // the GPU builder's scratch serves here too
        cudaStreamSynchronize(c->stream);
        dev_free(c, c->bld);
        if (!alloc(c->bld, bytes)) return TIM_RT_OK;
    }
    uint8_t* tmp = static_cast<uint8_t*>(c->bld.ptr);
    Ctl* ctl = reinterpret_cast<Ctl*>(tmp);
    uint32_t* parent = reinterpret_cast<uint32_t*>(tmp + o_par);
    uint32_t* arrivals = reinterpret_cast<uint32_t*>(tmp + o_arr);
    float4* cost = reinterpret_cast<float4*>(tmp + o_cost);
    uint32_t* item = reinterpret_cast<uint32_t*>(tmp + o_item);
    Box* item_e = reinterpret_cast<Box*>(tmp + o_e);
    uint2* base = reinterpret_cast<uint2*>(tmp + o_base);
    const In in{s->view.nodes, s->view.pleaf, n};
    cudaStream_t st = c->stream;
    Ctl h{};
    h.total = 1u;
    h.level[1] = 1u;
    const Box everything{{-FLT_MAX, -FLT_MAX, -FLT_MAX}, {FLT_MAX, FLT_MAX, FLT_MAX}};
    const uint32_t root = 0u, blocks = (n + 255u) / 256u;
    bool ok = cudaMemsetAsync(tmp, 0, bytes, st) == cudaSuccess &&
              cudaMemsetAsync(parent, 0xFF, 4ull * n, st) == cudaSuccess &&
              cudaMemcpyAsync(ctl, &h, sizeof(h), cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemcpyAsync(item, &root, 4, cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemcpyAsync(item_e, &everything, sizeof(Box), cudaMemcpyHostToDevice, st) == cudaSuccess;
    if (ok) {
        k_four_parents<<<blocks, 256, 0, st>>>(in, parent, ctl);
        k_four_cost<<<blocks, 256, 0, st>>>(in, parent, arrivals, cost, ctl);
        if (cap <= kSmallTree)
            k_four_small<<<1, 256, 0, st>>>(in, cost, item, item_e, base, cap, std::min<uint32_t>(s->depth, kMaxLevels), ctl);
        for (uint32_t lv = 0; cap > kSmallTree && lv < s->depth && lv < kMaxLevels; ++lv)
            k_four_level<<<std::min<uint32_t>(592u, (cap + 127u) / 128u), 128, 0, st>>>(in, cost, item, item_e, base, cap,
                                                                                        lv, ctl);
        ok = cudaGetLastError() == cudaSuccess &&
             cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
             cudaStreamSynchronize(st) == cudaSuccess;
    }
    uint32_t levels = 0;
    while (ok && levels < s->depth && h.level[levels + 1u] > h.level[levels]) ++levels;
    float bound[3];
    for (int d = 0; d < 3; ++d) memcpy(&bound[d], &h.bound[d], 4);
    const bool fits = ok && !h.bad && h.leaves && h.total <= kFourIndexMask && h.level[levels] == h.total && bound[0] <= 1.099511627776e12f &&
                      bound[1] <= 1.099511627776e12f && bound[2] <= 1.099511627776e12f;   // 2^40
    if (fits) {
        const uint64_t o_pairs = up((uint64_t)kFourBytes * h.total), o_leaf = o_pairs + up((uint64_t)kPairBytes * cap),
                       o_tri = o_leaf + up(32ull * h.leaves);
        if (alloc(s->trees, o_tri + 4ull * num_tris)) {
            uint8_t* t = static_cast<uint8_t*>(s->trees.ptr);
            SceneView& v = s->view;
            float4* nodes4 = reinterpret_cast<float4*>(t);
            float4* pairs = reinterpret_cast<float4*>(t + o_pairs);
            uint4* leaf4 = reinterpret_cast<uint4*>(t + o_leaf);
            uint32_t* tri_leaf4 = reinterpret_cast<uint32_t*>(t + o_tri);
            k_pairs<<<blocks, 256, 0, st>>>(in, pairs);
            Levels lv{levels, {}};
            std::copy(h.level, h.level + levels, lv.first);
            k_four_fill<<<(h.total + 127u) / 128u, 128, 0, st>>>(in, cost, item, item_e, base, h.total, lv, nodes4, leaf4,
                                                                 tri_leaf4);
            ok = cudaGetLastError() == cudaSuccess;
            v.nodes4 = nodes4;
            v.leaf4 = leaf4;
            v.tri_leaf4 = tri_leaf4;
            v.pairs = pairs;
            v.root_pair = root_left >> 1;
            v.depth4 = levels;
            for (int d = 0; d < 3; ++d) v.bound4[d] = bound[d];
        }
    }
    if (!ok) {
        set_error("building the 4-wide tree failed");
        return TIM_RT_EDEVICE;
    }
    return TIM_RT_OK;
}

}  // namespace timrt
