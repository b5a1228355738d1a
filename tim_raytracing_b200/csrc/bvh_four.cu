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
// form does the same on the host; here it is a few short kernels (and one launch a level in
// large trees) that run while the host brings the vertices over, or, in the smallest
// scenes, the host's own work: there the kernels' latencies were most of an upload
// (kHostTree has figures).
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <string>
#include "common.cuh"
#include "context.h"
#include "four_stack.h"
#include "kernels.h"

namespace timrt {

TreePlan::TreePlan(uint64_t nodes4, uint64_t inner, uint64_t leaves, uint64_t tris)
    : pairs(up256(kFourBytes * nodes4)), leaf4(pairs + up256(kPairBytes * inner)), tri_leaf4(leaf4 + up256(32ull * leaves)),
      bytes(tri_leaf4 + 4ull * tris) {}

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
    const float4* nodes;     // on the host of any alignment
    const uint4* pleaf;      // per node: (first triangle, leaf header, ...)
    uint32_t num_nodes;
};

__host__ __device__ __forceinline__ float4 node_vec(const In& in, uint32_t k) {
#ifdef __CUDA_ARCH__
    return in.nodes[k];
#else
    float4 v;
    std::memcpy(&v, in.nodes + k, sizeof(v));
    return v;
#endif
}
__host__ __device__ __forceinline__ uint32_t bits_of(float v) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(v);
#else
    uint32_t b;
    std::memcpy(&b, &v, 4);
    return b;
#endif
}
__host__ __device__ __forceinline__ float float_of(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float v;
    std::memcpy(&v, &b, 4);
    return v;
#endif
}

struct Box { float lo[3], hi[3]; };

// Least and largest of two numbers (the host compiler calls a function for fminf).
__host__ __device__ __forceinline__ float least(float a, float b) {
#ifdef __CUDA_ARCH__
    return fminf(a, b);
#else
    return b < a ? b : a;
#endif
}
__host__ __device__ __forceinline__ float largest(float a, float b) {
#ifdef __CUDA_ARCH__
    return fmaxf(a, b);
#else
    return a < b ? b : a;
#endif
}

// A subtree on its way into a slot: node id | leaf bit, slots it may take, its stored
// box and the intersection E of that box and its ancestors'.
struct Sub {
    uint32_t id;
    int k;
    Box box, e;
};

__host__ __device__ __forceinline__ uint32_t children_of(const In& in, uint32_t x) {
    uint32_t c;
#ifdef __CUDA_ARCH__
    c = reinterpret_cast<const uint4*>(in.nodes + 4u * x)->z;
#else
    std::memcpy(&c, reinterpret_cast<const uint8_t*>(in.nodes + 4u * x) + 8, 4);
#endif
    return c;
}

__host__ __device__ __forceinline__ void child_boxes(const In& in, uint32_t x, Box& l, Box& r) {
    const float4 a = node_vec(in, 4u * x + 1u), b = node_vec(in, 4u * x + 2u), c = node_vec(in, 4u * x + 3u);
    const float la[6] = {a.x, a.y, c.x, a.z, a.w, c.y}, ra[6] = {b.x, b.y, c.z, b.z, b.w, c.w};
    for (int d = 0; d < 3; ++d) {   // the slab test orders each axis itself
        l.lo[d] = least(la[d], la[3 + d]); l.hi[d] = largest(la[d], la[3 + d]);
        r.lo[d] = least(ra[d], ra[3 + d]); r.hi[d] = largest(ra[d], ra[3 + d]);
    }
}

__host__ __device__ __forceinline__ uint32_t left_id(uint32_t packed) {
    return (packed & kNidMask) | (packed & kNidLeftLeafBit ? kNidLeafBit : 0u);
}
__host__ __device__ __forceinline__ uint32_t right_id(uint32_t packed) {
    return ((packed & kNidMask) + 1u) | (packed & kNidRightLeafBit ? kNidLeafBit : 0u);
}

__host__ __device__ __forceinline__ float area_of(const Box& b) {
    const float x = b.hi[0] - b.lo[0], y = b.hi[1] - b.lo[1], z = b.hi[2] - b.lo[2];
    return x * y + y * z + z * x;
}

// Least cost of covering a subtree with at most k = 0..4 slots. Leaves cost nothing
// (every cut of the tree holds all of them); a subtree without triangles takes no slot.
struct Cover { float f[5]; };

__host__ __device__ __forceinline__ Cover cover_of(const In& in, const float4* cost, uint32_t id) {
    Cover c;
    const uint32_t x = id & kNidMask;
    if (id & kNidLeafBit) {
        const bool empty = (in.pleaf[x].y & ((1u << kTriBits) - 1u)) == 0u;
        c.f[0] = empty ? 0.0f : INFINITY;
        c.f[1] = c.f[2] = c.f[3] = c.f[4] = 0.0f;
        return c;
    }
#ifdef __CUDA_ARCH__
    const float4 v = __ldcg(cost + x);
#else
    const float4 v = cost[x];
#endif
    const bool empty = v.x < 0.0f;
    c.f[0] = empty ? 0.0f : INFINITY;
    c.f[1] = empty ? 0.0f : v.x;
    c.f[2] = empty ? 0.0f : v.y;
    c.f[3] = empty ? 0.0f : v.z;
    c.f[4] = empty ? 0.0f : v.w;
    return c;
}

// Best division of k slots between two subtrees: the cost, and the left one's share.
__host__ __device__ __forceinline__ float divide(const Cover& l, const Cover& r, int k, int& share) {
    float best = INFINITY;
    share = 0;
#pragma unroll
    for (int j = 0; j <= 4; ++j) {
        if (j > k) break;
        const float v = l.f[j] + r.f[k - j];
        if (v < best) { best = v; share = j; }
    }
    return best;
}

// An inner node's costs, and what they stand for: per number of slots k = 1 to 4, at bits
// 4 (k - 1) and up, the left child's share of them and, above it, whether the node is
// divided at all (it takes one slot otherwise); kHasTris unless no triangle is below. Made
// here once, so that the numbering of the nodes reads one word a subtree: with both
// children's costs and three divisions for each, a level of it took 13 to 23 us.
constexpr uint32_t kHasTris = 1u << 16;
struct NodeCost { float4 cost; uint32_t plan; };

// Of an inner node with these children; area: its own box's.
__host__ __device__ __forceinline__ NodeCost cost_of(const In& in, const float4* cost, uint32_t packed, float area) {
    const Cover l = cover_of(in, cost, left_id(packed)), r = cover_of(in, cost, right_id(packed));
    if (l.f[0] == 0.0f && r.f[0] == 0.0f) return {make_float4(-1.0f, 0.0f, 0.0f, 0.0f), 0u};   // no triangle below
    float d[5];
    int share[5];
    for (int k = 1; k <= 4; ++k) {
        d[k] = divide(l, r, k, share[k]);
        if (r.f[0] == 0.0f) share[k] = k;   // no slot goes to a subtree without triangles (on the left none does)
    }
    const float single = area + d[4];
    uint32_t plan = kHasTris;
    for (int k = 1; k <= 4; ++k) plan |= ((uint32_t)share[k] | (d[k] < single ? 8u : 0u)) << (4 * (k - 1));
    return {make_float4(least(single, d[1]), least(single, d[2]), least(single, d[3]), least(single, d[4])), plan};
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
__global__ void k_four_cost(In in, const uint32_t* parent, uint32_t* arrivals, float4* cost, uint32_t* plan, const Ctl* ctl) {
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
        const uint32_t pp = parent[p];
        uint32_t up = 0;
        float area = 0.0f;
        if (pp != kNone) {
            up = children_of(in, pp);
            Box a, b;
            child_boxes(in, pp, a, b);
            area = area_of(p == (up & kNidMask) ? a : b);
        }
        const NodeCost v = cost_of(in, cost, packed, area);
        __stcg(cost + p, v.cost);
        plan[p] = v.plan;
        if (pp == kNone) return;
        if ((p == (up & kNidMask) ? left_id(up) : right_id(up)) & kNidLeafBit) return;   // used as a leaf above
        p = pp;
        packed = up;
    }
}

// The slots of the 4-wide node of binary node x (at most 4; leaves without triangles
// take none), by increasing area: the walk takes the last slot it entered first, and the largest is the likeliest occluder.
struct Slots {
    Sub sub[4];
    int n;
    uint32_t order;   // two bits each: the place in sub of the k-th by area
    __host__ __device__ __forceinline__ const Sub& operator[](int k) const { return sub[order >> (2 * k) & 3u]; }
};
__host__ __device__ __forceinline__ void expand(const In& in, const uint32_t* plan, uint32_t x, const Box& e, Slots& out) {
    Sub st[4];   // the shares of the subtrees on it never sum to more than four
    float area[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    int sp = 0, n = 0;
    auto push = [&](uint32_t node, uint32_t word, int k, const Box& pe) {
        const uint32_t packed = children_of(in, node);
        Sub a, b;
        a.id = left_id(packed);
        b.id = right_id(packed);
        child_boxes(in, node, a.box, b.box);
        a.k = (int)(word >> (4 * (k - 1)) & 7u);
        b.k = k - a.k;
        for (Sub* c : {&a, &b})
            for (int d = 0; d < 3; ++d) {
                c->e.lo[d] = largest(pe.lo[d], c->box.lo[d]);
                c->e.hi[d] = least(pe.hi[d], c->box.hi[d]);
            }
        if (b.k) st[sp++] = b;   // a subtree without triangles takes no slot
        if (a.k) st[sp++] = a;
    };
    if (plan[x] & kHasTris) push(x, plan[x], 4, e);   // only a root has none
    while (sp > 0) {
        const Sub s = st[--sp];
        if (!(s.id & kNidLeafBit)) {
            const uint32_t word = plan[s.id];
            if (word >> (4 * (s.k - 1)) & 8u) {
                push(s.id, word, s.k, s.e);
                continue;
            }
        }
        const float v = area_of(s.box);
        area[0] = n == 0 ? v : area[0];
        area[1] = n == 1 ? v : area[1];
        area[2] = n == 2 ? v : area[2];
        area[3] = n == 3 ? v : area[3];
        out.sub[n++] = s;
    }
    out.n = n;
    out.order = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        int rank = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) rank += j < n && (area[j] < area[i] || (area[j] == area[i] && j < i)) ? 1 : 0;
        if (i < n) out.order |= (uint32_t)i << (2 * rank);
    }
}

// Node w of a level: its inner slots become nodes of the next one.
__device__ void four_node(const In& in, const uint32_t* plan, uint32_t* item, Box* item_e, uint2* base, uint32_t cap, uint32_t w,
                          Ctl* ctl) {
    Slots s;
    expand(in, plan, item[w], item_e[w], s);
    const int n = s.n;
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

__global__ void __launch_bounds__(128) k_four_level(In in, const uint32_t* plan, uint32_t* item, Box* item_e, uint2* base,
                                                    uint32_t cap, uint32_t lv, Ctl* ctl) {
    if (!ctl->bad) {
        const uint32_t end = ctl->level[lv + 1u];
        for (uint32_t w = ctl->level[lv] + blockIdx.x * blockDim.x + threadIdx.x; w < end; w += gridDim.x * blockDim.x)
            four_node(in, plan, item, item_e, base, cap, w, ctl);
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
// of which half are empty: 47 us for 2,621 nodes (55 with its counters in global memory),
// where a launch takes 8 to 13 us, an empty one 4. With 3,300 inner nodes an upload took as
// long either way.
constexpr uint32_t kSmallTree = 2048u, kSmallThreads = 512u;   // inner binary nodes
__global__ void __launch_bounds__(kSmallThreads) k_four_small(In in, const uint32_t* plan, uint32_t* item, Box* item_e, uint2* base,
                                                    uint32_t cap, uint32_t depth, Ctl* ctl) {
    __shared__ Ctl c;   // the counters of the block's levels
    if (threadIdx.x == 0) c = *ctl;
    __syncthreads();
    uint32_t begin = 0u, end = 1u;
    for (uint32_t lv = 0; lv < depth && begin < end; ++lv) {
        if (!c.bad)
            for (uint32_t w = begin + threadIdx.x; w < end; w += blockDim.x) four_node(in, plan, item, item_e, base, cap, w, &c);
        __syncthreads();
        begin = end;
        end = c.total;
        if (threadIdx.x == 0) c.level[lv + 2u] = end;
        __syncthreads();
    }
    if (threadIdx.x == 0) *ctl = c;
}

// The first node of each level.
struct Levels { uint32_t count, first[kMaxLevels]; };

// Node w of the slots s, whose inner slots' nodes are numbered from b.x on and whose leaves'
// records from b.y; below: the levels after w's.
__host__ __device__ __forceinline__ void fill_node(const In& in, uint32_t w, const Slots& s, uint2 b, uint32_t below,
                                                   float4* nodes4, uint4* leaf4, uint32_t* tri_leaf4) {
    float lo[3][4], hi[3][4];
    uint32_t ref[4];
    const int n = s.n;
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
        leaf4[2u * b.y] = make_uint4(bits_of(e.lo[0]), bits_of(e.lo[1]), bits_of(e.lo[2]), nid);
        leaf4[2u * b.y + 1u] = make_uint4(bits_of(e.hi[0]), bits_of(e.hi[1]), bits_of(e.hi[2]), (empty ? 2u : 0u) | nt << 2);
        for (uint32_t t = 0; t < nt; ++t) tri_leaf4[li.x + t] = b.y;
        ++b.y;
    }
    float4* o = nodes4 + (kFourBytes / 16u) * (uint64_t)w;
    for (uint32_t d = 0; d < 3u; ++d) {
        o[4u * d] = o[4u * d + 3u] = make_float4(lo[d][0], lo[d][1], lo[d][2], lo[d][3]);
        o[4u * d + 1u] = o[4u * d + 2u] = make_float4(hi[d][0], hi[d][1], hi[d][2], hi[d][3]);
    }
    o[12] = make_float4(float_of(ref[0]), float_of(ref[1]), float_of(ref[2]), float_of(ref[3]));
    o[13] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The record of each inner node's children (trace_pair.cuh), at half the left one's id.
__host__ __device__ __forceinline__ void fill_pair(const In& in, uint32_t i, float4* pairs) {
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
    o[6] = make_float4(float_of(ref[0]), float_of(ref[1]), 0.f, 0.f);
}

// The nodes of the 4-wide tree, by the first blocks, and the records of child pairs.
__global__ void __launch_bounds__(128) k_four_fill(In in, const uint32_t* plan, const uint32_t* item, const Box* item_e,
                                                   const uint2* base, uint32_t total, Levels levels, float4* nodes4,
                                                   uint4* leaf4, uint32_t* tri_leaf4, float4* pairs) {
    const uint32_t node_blocks = (total + 127u) / 128u;
    if (blockIdx.x >= node_blocks) {
        const uint32_t i = (blockIdx.x - node_blocks) * 128u + threadIdx.x;
        if (i < in.num_nodes) fill_pair(in, i, pairs);
        return;
    }
    const uint32_t w = blockIdx.x * 128u + threadIdx.x;
    if (w >= total) return;
    uint32_t below = 0;   // the levels after w's
    for (uint32_t lv = 1; lv < levels.count; ++lv) below += w < levels.first[lv] ? 1u : 0u;
    Slots s;
    expand(in, plan, item[w], item_e[w], s);
    fill_node(in, w, s, base[w], below, nodes4, leaf4, tri_leaf4);
}

// Per node (first triangle, leaf header, leaf-data offset, 0); a node without leaf data
// (offset 0xFFFFFFFF) gets header 0, as the kernels read it; node 0's last word is left
// with the number of triangles. A block takes the places of its nodes' triangles together,
// blocks in any order: nothing depends on it, and it may differ from upload to upload. The
// trees' build starts here too (work): its counters, its first item, parents and arrivals.
struct Work {
    Ctl* ctl;
    uint32_t *parent, *arrivals, *item, *plan;
    float4* cost;
    Box* item_e;
    uint2* base;
};
__global__ void __launch_bounds__(256) k_leaf_info(const float4* nodes, const uint32_t* leaf, uint32_t n, uint4* info,
                                                   Work work) {
    __shared__ uint32_t warp_sum[8], block_base;
    const uint32_t i = blockIdx.x * 256u + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (work.ctl && i < n) {
        work.parent[i] = kNone;
        work.arrivals[i] = 0u;
        if (i == 0u) {
            Ctl c{};
            c.total = 1u;
            c.level[1] = 1u;
            *work.ctl = c;
            work.item[0] = 0u;
            for (int d = 0; d < 3; ++d) {
                work.item_e->lo[d] = -FLT_MAX;
                work.item_e->hi[d] = FLT_MAX;
            }
        }
    }
    uint32_t off = 0xFFFFFFFFu, hdr = 0u;
    if (i < n) {
        off = reinterpret_cast<const uint4*>(nodes + 4u * i)->w;
        hdr = off == 0xFFFFFFFFu ? 0u : leaf[off];
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
    info[i].x = block_base + warp_sum[warp] + sum - nt;
    info[i].y = hdr;
    info[i].z = off;
    if (i) info[i].w = 0u;
}

// Per leaf-data triangle record, in its leaf's order: (p0, vertexOffset) (p1 - p0, index01)
// (p2 - p0, index2_matId), the edges being the same rounded differences CollideTriangle
// forms (collision.glsl:60-61). Runs after validate_bvh, so every offset and vertex index is
// in range. The host loop this replaces and the copy of its result were half of a
// 1M-triangle scene's upload.
__global__ void __launch_bounds__(256) k_leaf_tris(const uint32_t* leaf, const float* pos, uint32_t n, const uint4* info,
                                                   float4* tris) {
    const uint32_t i = blockIdx.x * 256u + threadIdx.x;
    if (i >= n) return;
    const uint4 li = info[i];
    const uint32_t nt = li.y & ((1u << kTriBits) - 1u);
    for (uint32_t t = 0; t < nt; ++t) {
        const uint32_t* r = leaf + 1u + li.z + 3u * t;
        const uint32_t r0 = r[0], r1 = r[1], r2 = r[2];
        const float* P0 = pos + 3ull * (r0 + (r1 & 0xFFFFu));
        const float* P1 = pos + 3ull * (r0 + (r1 >> 16));
        const float* P2 = pos + 3ull * (r0 + (r2 & 0xFFFFu));
        float4* o = tris + 3ull * (li.x + t);
        o[0] = make_float4(P0[0], P0[1], P0[2], __uint_as_float(r0));
        o[1] = make_float4(P1[0] - P0[0], P1[1] - P0[1], P1[2] - P0[2], __uint_as_float(r1));
        o[2] = make_float4(P2[0] - P0[0], P2[1] - P0[1], P2[2] - P0[2], __uint_as_float(r2));
    }
}

// Whether a scene can have the trees at all. With a memory budget it keeps to the arrays it
// always had, so that what was admitted stays admitted; BLAS boxes are tested by the binary
// walk only.
bool wants_trees(const tim_rt_ctx* c, uint32_t n, uint32_t num_blas, uint64_t tris) {
    return !c->budget && !num_blas && n >= 2u && tris && tris < kFourFirstMask;
}

constexpr float kMostPlane = 1.099511627776e12f;   // 2^40: the any-hit box test's bounds

void set_trees(SceneView& v, const uint8_t* t, const TreePlan& p, uint32_t root_left, uint32_t levels, const float bound[3]) {
    v.nodes4 = reinterpret_cast<const float4*>(t);
    v.pairs = reinterpret_cast<const float4*>(t + p.pairs);
    v.leaf4 = reinterpret_cast<const uint4*>(t + p.leaf4);
    v.tri_leaf4 = reinterpret_cast<const uint32_t*>(t + p.tri_leaf4);
    v.root_pair = root_left >> 1;
    v.depth4 = levels;
    for (int d = 0; d < 3; ++d) v.bound4[d] = bound[d];
}

}  // namespace

cudaError_t fill_leaf_tris(const Scene* s, cudaStream_t stream) {
    const uint32_t n = s->pc.numNodes;
    k_leaf_tris<<<(n + 255u) / 256u, 256, 0, stream>>>(s->view.leaf, s->view.pos, n, s->view.pleaf,
                                                      const_cast<float4*>(s->view.ptris));
    return cudaGetLastError();
}

cudaError_t TreeBuild::begin() {
    const uint32_t n = s->pc.numNodes;
    Work w{};
    cap = n / 2u + 1u;   // inner nodes
    if (wants_trees(c, n, s->pc.numBlas, num_tris)) {
        const uint64_t o_par = up256(sizeof(Ctl)), o_arr = o_par + up256(4ull * n), o_plan = o_arr + up256(4ull * n),
                       o_cost = o_plan + up256(4ull * n), o_item = o_cost + up256(16ull * n), o_e = o_item + up256(4ull * cap),
                       o_base = o_e + up256(sizeof(Box) * cap), bytes = o_base + up256(8ull * cap);
        // The scratch lies where the leaf triangles come in the end, which is enough but for
        // trees of fewer than two triangles a leaf; no room for them is no error: the plain
        // walk stays.
        tmp = static_cast<uint8_t*>(s->ptris.ptr);
        if (s->ptris.bytes < bytes) {
            const std::string last_error = tim_rt_last_error();
            tmp = nullptr;
            if (dev_alloc(c, scratch, bytes) == TIM_RT_OK) tmp = static_cast<uint8_t*>(scratch.ptr);
            else set_error(last_error);
        }
        if (tmp)
            w = Work{reinterpret_cast<Ctl*>(tmp),
                     reinterpret_cast<uint32_t*>(tmp + o_par),
                     reinterpret_cast<uint32_t*>(tmp + o_arr),
                     reinterpret_cast<uint32_t*>(tmp + o_item),
                     reinterpret_cast<uint32_t*>(tmp + o_plan),
                     reinterpret_cast<float4*>(tmp + o_cost),
                     reinterpret_cast<Box*>(tmp + o_e),
                     reinterpret_cast<uint2*>(tmp + o_base)};
        o[0] = o_plan; o[1] = o_item; o[2] = o_e; o[3] = o_base;
    }
    cudaStream_t st = c->stream;
    const uint32_t blocks = (n + 255u) / 256u;
    uint4* info = const_cast<uint4*>(s->view.pleaf);
    cudaMemsetAsync(info, 0, 16, st);   // node 0's last word counts the triangles handed out
    k_leaf_info<<<blocks, 256, 0, st>>>(s->view.nodes, s->view.leaf, n, info, w);
    if (tmp) {
        const In in{s->view.nodes, s->view.pleaf, n};
        k_four_parents<<<blocks, 256, 0, st>>>(in, w.parent, w.ctl);
        k_four_cost<<<blocks, 256, 0, st>>>(in, w.parent, w.arrivals, w.cost, w.plan, w.ctl);
        if (cap <= kSmallTree)
            k_four_small<<<1, kSmallThreads, 0, st>>>(in, w.plan, w.item, w.item_e, w.base, cap,
                                                      std::min<uint32_t>(s->depth, kMaxLevels), w.ctl);
        for (uint32_t lv = 0; cap > kSmallTree && lv < s->depth && lv < kMaxLevels; ++lv)
            k_four_level<<<std::min<uint32_t>(592u, (cap + 127u) / 128u), 128, 0, st>>>(in, w.plan, w.item, w.item_e, w.base,
                                                                                        cap, lv, w.ctl);
    }
    return cudaGetLastError();
}

int TreeBuild::end(uint32_t root_left) {
    if (!tmp) return TIM_RT_OK;
    const uint32_t n = s->pc.numNodes;
    cudaStream_t st = c->stream;
    Ctl h{};
    bool ok = cudaMemcpyAsync(&h, tmp, sizeof(h), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
              cudaStreamSynchronize(st) == cudaSuccess;
    uint32_t levels = 0;
    while (ok && levels < s->depth && h.level[levels + 1u] > h.level[levels]) ++levels;
    float bound[3];
    for (int d = 0; d < 3; ++d) memcpy(&bound[d], &h.bound[d], 4);
    if (ok && !h.bad && h.leaves && h.total <= kFourIndexMask && h.level[levels] == h.total && bound[0] <= kMostPlane &&
        bound[1] <= kMostPlane && bound[2] <= kMostPlane) {
        const TreePlan p(h.total, cap, h.leaves, num_tris);
        const std::string last_error = tim_rt_last_error();
        if (dev_alloc(c, s->trees, p.bytes) == TIM_RT_OK) {
            uint8_t* t = static_cast<uint8_t*>(s->trees.ptr);
            const In in{s->view.nodes, s->view.pleaf, n};
            Levels lv{levels, {}};
            std::copy(h.level, h.level + levels, lv.first);
            k_four_fill<<<(h.total + 127u) / 128u + (n + 127u) / 128u, 128, 0, st>>>(
                in, reinterpret_cast<uint32_t*>(tmp + o[0]), reinterpret_cast<uint32_t*>(tmp + o[1]), reinterpret_cast<Box*>(tmp + o[2]),
                reinterpret_cast<uint2*>(tmp + o[3]), h.total, lv, reinterpret_cast<float4*>(t),
                reinterpret_cast<uint4*>(t + p.leaf4), reinterpret_cast<uint32_t*>(t + p.tri_leaf4),
                reinterpret_cast<float4*>(t + p.pairs));
            ok = cudaGetLastError() == cudaSuccess;
            set_trees(s->view, t, p, root_left, levels, bound);
        } else {
            set_error(last_error);
        }
    }
    if (!ok) {
        set_error("building the 4-wide tree failed");
        return TIM_RT_EDEVICE;
    }
    return TIM_RT_OK;
}

TreeBuild::~TreeBuild() { dev_free(c, scratch); }   // waits for the kernels that use it

// ------------------------------------------------------------------- the smallest scenes

namespace {

// Nodes up to which the host makes the trees: the whole upload by the host / by the kernels,
// 63 nodes 0.043 / 0.13 ms, 651 0.084 / 0.12, 863 0.09 / 0.18, 2,015 0.196 / 0.169, 2,621
// 0.28 / 0.185. The host takes 50 ns a node, the kernels' latencies 100 us and more.
constexpr uint32_t kHostTree = 1536u;

}  // namespace

bool host_trees(const tim_rt_ctx* c, const uint8_t* blob, const uint32_t ranges[7][2], const tim_rt_push_constants& pc,
                uint32_t depth, uint64_t tris, HostTrees& out) {
    const uint32_t n = pc.numNodes;
    if (n > kHostTree || !wants_trees(c, n, pc.numBlas, tris)) return false;
    const float4* nodes = reinterpret_cast<const float4*>(blob + ranges[TIM_RT_RANGE_NODE][0]);
    const uint8_t* leaf = blob + ranges[TIM_RT_RANGE_LEAF][0];
    std::vector<uint4> info(n);
    std::vector<uint32_t> parent(n, kNone);
    std::vector<float4> cost(n);
    std::vector<uint32_t> plan(n);
    const In in{nodes, info.data(), n};
    float bound[3] = {0.f, 0.f, 0.f};
    uint32_t first = 0;
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t off, hdr = 0u;
        std::memcpy(&off, reinterpret_cast<const uint8_t*>(nodes + 4u * i) + 12, 4);
        if (off != 0xFFFFFFFFu) std::memcpy(&hdr, leaf + 4ull * off, 4);
        info[i] = make_uint4(first, hdr, off, 0u);
        first += hdr & ((1u << kTriBits) - 1u);
        const uint32_t l = children_of(in, i) & kNidMask;
        if (l == kNidMask) continue;
        if (parent[l] != kNone || parent[l + 1u] != kNone) return false;   // a shared child
        parent[l] = parent[l + 1u] = i;
        for (uint32_t w = 1; w < 4u; ++w) {
            const float4 v = node_vec(in, 4u * i + w);
            if (!(std::isfinite(v.x) && std::isfinite(v.y) && std::isfinite(v.z) && std::isfinite(v.w))) return false;
        }
        Box b[2];
        child_boxes(in, i, b[0], b[1]);
        for (const Box& x : b)
            for (int d = 0; d < 3; ++d) bound[d] = std::max(bound[d], std::max(std::fabs(x.lo[d]), std::fabs(x.hi[d])));
    }
    if (!(bound[0] <= kMostPlane && bound[1] <= kMostPlane && bound[2] <= kMostPlane)) return false;
    for (uint32_t i = n; i-- > 0u;) {   // children have higher ids
        const uint32_t packed = children_of(in, i), p = parent[i];
        if ((packed & kNidMask) == kNidMask) continue;
        float area = 0.0f;
        if (p != kNone) {
            Box a, b;
            child_boxes(in, p, a, b);
            area = area_of(i == (children_of(in, p) & kNidMask) ? a : b);
        }
        const NodeCost v = cost_of(in, cost.data(), packed, area);
        cost[i] = v.cost;
        plan[i] = v.plan;
    }
    struct Node { uint32_t item; Box e; Slots s; uint2 base; };
    std::vector<Node> q(1);
    q[0].item = 0u;
    for (int d = 0; d < 3; ++d) { q[0].e.lo[d] = -FLT_MAX; q[0].e.hi[d] = FLT_MAX; }
    q.reserve(n / 2u + 1u);
    std::vector<uint32_t> level{0u};   // the first node of each
    uint32_t leaves = 0;
    for (uint32_t w = 0, end = 1u; w < q.size(); ++w) {
        if (w == end) {
            level.push_back(w);
            end = (uint32_t)q.size();
        }
        expand(in, plan.data(), q[w].item, q[w].e, q[w].s);
        q[w].base = make_uint2((uint32_t)q.size(), leaves);
        for (int k = 0; k < q[w].s.n; ++k) {
            const Sub sub = q[w].s[k];
            if (sub.id & kNidLeafBit) {
                ++leaves;
                continue;
            }
            if (q.size() > n / 2u) return false;
            q.emplace_back();
            q.back().item = sub.id;
            q.back().e = sub.e;
        }
    }
    if (!leaves || level.size() > depth) return false;
    const TreePlan p(q.size(), n / 2u + 1u, leaves, tris);
    out.trees_at = up256(16ull * n);
    out.image.resize(out.trees_at + p.bytes);
    std::memcpy(out.image.data(), info.data(), 16ull * n);
    uint8_t* t = out.image.data() + out.trees_at;
    for (uint32_t w = 0, lv = 0; w < q.size(); ++w) {
        if (lv + 1u < level.size() && w == level[lv + 1u]) ++lv;
        fill_node(in, w, q[w].s, q[w].base, (uint32_t)level.size() - 1u - lv, reinterpret_cast<float4*>(t),
                  reinterpret_cast<uint4*>(t + p.leaf4), reinterpret_cast<uint32_t*>(t + p.tri_leaf4));
    }
    for (uint32_t i = 0; i < n; ++i) fill_pair(in, i, reinterpret_cast<float4*>(t + p.pairs));
    out.plan = p;
    out.levels = (uint32_t)level.size();
    std::copy(bound, bound + 3, out.bound);
    return true;
}

void HostTrees::place(const uint8_t* d, uint32_t root_left, SceneView& v) const {
    v.pleaf = reinterpret_cast<const uint4*>(d);
    set_trees(v, d + trees_at, plan, root_left, levels, bound);
}

}  // namespace timrt
