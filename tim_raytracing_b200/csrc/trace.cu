// trace.cu -- persistent ray-tracing kernels for sm_100a and their launchers.
//
// Every trace kernel here is the same persistent loop: a grid sized to fill
// the GPU (blocks per SM from the occupancy calculator x 148 SMs), in which
// each warp keeps all 32 lanes busy by refilling finished lanes with new work
// items from a global atomic counter (one atomicAdd per refill, issued by one
// elected lane). A policy object turns a work item into a ray (load) and
// writes the result (store): plain ray batches, camera pixels, secondary
// (shadow / probe-visibility / bounce) rays.
//
// Coherence: camera work items walk the frame in 8x4-pixel tiles (32 pixels =
// one warp), and the secondary rays of those pixels are queued by kind -- sun,
// tile-light slot j, probe corner i, bounce -- in one segment per kind, so a
// warp traces 32 rays of the same kind from neighbouring pixels.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdio>
#include "common.cuh"
#include "trace_plain.cuh"
#include "trace_wide.cuh"
#include "walk.cuh"
#include "kernels.h"
#include "../../include/tim_rt.h"

namespace timrt {

// Secondary-ray kinds, one queue segment each.
constexpr uint32_t kKindSun = 0, kKindLight0 = 1, kKindProbe0 = 17, kKindBounce = 25, kNumKinds = 26;

// The secondary queue split into bands of output rows (one band unless a camera
// trace is pipelined): band b's rays of kind k take cap[b] slots from
// base[b] + k * cap[b]; its counts and prefix entries are b * kNumKinds + k.
struct QueueBands {
    uint32_t n;
    uint32_t row[kMaxCamBands + 1];   // band b: output rows [row[b], row[b + 1])
    uint32_t base[kMaxCamBands];
    uint32_t cap[kMaxCamBands];
};

__device__ __forceinline__ uint32_t band_of_row(const QueueBands& q, uint32_t r) {
    uint32_t b = 0;
    for (uint32_t k = 1; k < q.n; ++k) b += r >= q.row[k] ? 1u : 0u;
    return b;
}

// Work item -> pixel in 8x4 tiles (row-major tiles over the frame).
__device__ __forceinline__ bool tile_pixel(uint32_t i, uint32_t W, uint32_t H, uint32_t& px, uint32_t& py) {
    const uint32_t tiles_x = (W + 7u) >> 3;
    const uint32_t tile = i >> 5, within = i & 31u;
    px = (tile % tiles_x) * 8u + (within & 7u);
    py = (tile / tiles_x) * 4u + (within >> 3);
    return px < W && py < H;
}

__host__ __device__ __forceinline__ uint32_t tiled_work_items(uint32_t W, uint32_t H) {
    return ((W + 7u) >> 3) * ((H + 3u) >> 2) * 32u;
}

// -------------------------------------------------------------------- policies

// The leaf kind a policy's rays take (kLeafOne unless the policy says otherwise).
template <class P, class = void>
struct leaf_kind { static constexpr int value = kLeafOne; };
template <class P>
struct leaf_kind<P, decltype((void)P::kLeaf)> { static constexpr int value = P::kLeaf; };
struct BatchPolicy {
    const tim_rt_ray* rays;
    uint4* hit;
    uint32_t* nid;
    float2* bary;
    uint32_t mode;

    __device__ __forceinline__ bool load(const SceneView&, uint32_t i, TravState& st) const {
        const float4* rp = reinterpret_cast<const float4*>(rays + i);
        const float4 a = __ldg(rp), b = __ldg(rp + 1);
        st.r.ox = a.x; st.r.oy = a.y; st.r.oz = a.z;
        st.r.dx = b.x; st.r.dy = b.y; st.r.dz = b.z;
        st.t = a.w;
        const uint32_t fl = __float_as_uint(b.w);
        st.any = (mode == TIM_RT_MODE_ANY) || (mode == TIM_RT_MODE_PER_RAY && (fl & TIM_RT_RAY_ANY));
        st.dup_ok = nid == nullptr;
        return true;
    }
    __device__ __forceinline__ void store(const SceneView&, uint32_t i, const TravState& st, float tmax0) const {
        if (st.any) {
            hit[i] = make_uint4(st.hit ? 1u : 0u, 0u, 0u, __float_as_uint(tmax0));
            if (nid) nid[i] = 0xFFFFFFFFu;
            if (bary) bary[i] = make_float2(0.f, 0.f);
        } else {
            hit[i] = make_uint4(st.rec0, st.rec1, st.rec2, __float_as_uint(st.t));
            if (nid) nid[i] = st.hit ? st.nid : 0xFFFFFFFFu;
            if (bary) bary[i] = make_float2(st.u, st.v);
        }
    }
    __device__ __forceinline__ void skip(uint32_t) const {}
    __device__ __forceinline__ bool wants_nid(const TravState&) const { return nid != nullptr; }
    __device__ __forceinline__ bool wants_bary(const TravState&) const { return bary != nullptr; }
};

// The rays of one kind of a TIM_RT_MODE_PER_RAY batch: the two kinds walk different
// trees, each in a launch of its own.
struct KindBatchPolicy : BatchPolicy {
    static constexpr bool kFilters = true;
    uint32_t kind;   // TIM_RT_RAY_ANY or 0
    __device__ __forceinline__ bool keeps(uint32_t i) const {
        return (__ldg(reinterpret_cast<const uint32_t*>(rays + i) + 7) & TIM_RT_RAY_ANY) == kind;
    }
};

// Any-hit rays of a two-level scene (TIM_RT_TRACE_TLAS): traverseTlasFast
// (bvhTraversal_inline.glsl:83-151 with TLAS_COLLIDE) from the scene root.
struct TlasBatchPolicy : BatchPolicy {
    static constexpr int kLeaf = kLeafTlasTop;
};

// cameraPass.comp:44-76 pinhole ray of invocation (gx, gy) (cameraPass.comp:50-54).
__device__ __forceinline__ void camera_ray(const tim_rt_pass_data& pd, uint32_t gx, uint32_t gy, float& dx, float& dy,
                                           float& dz) {
    const float fx = (float)gx, fy = (float)gy;
    const float swx = (pd.frustumCorner10[0] - pd.frustumCorner00[0]) * pd.invFrameSize[0];
    const float swy = (pd.frustumCorner10[1] - pd.frustumCorner00[1]) * pd.invFrameSize[0];
    const float swz = (pd.frustumCorner10[2] - pd.frustumCorner00[2]) * pd.invFrameSize[0];
    const float shx = (pd.frustumCorner01[0] - pd.frustumCorner00[0]) * pd.invFrameSize[1];
    const float shy = (pd.frustumCorner01[1] - pd.frustumCorner00[1]) * pd.invFrameSize[1];
    const float shz = (pd.frustumCorner01[2] - pd.frustumCorner00[2]) * pd.invFrameSize[1];
    const float tx = (pd.frustumCorner00[0] + swx * fx) + shx * fy;
    const float ty = (pd.frustumCorner00[1] + swy * fx) + shy * fy;
    const float tz = (pd.frustumCorner00[2] + swz * fx) + shz * fy;
    const float vx = tx - pd.cameraPos[0], vy = ty - pd.cameraPos[1], vz = tz - pd.cameraPos[2];
    const float len = sqrtf(dot3(vx, vy, vz, vx, vy, vz));   // normalize(v) = v / sqrt(dot(v, v))
    dx = vx / len;
    dy = vy / len;
    dz = vz / len;
}

// One work item per pixel, tile order. Output row py is traced by invocation
// gy = 16*ceil(H/16) - py (cameraPass.comp:46), so row 0 is never traced.
struct CameraPolicy {
    tim_rt_pass_data pd;
    uint32_t ngy16;         // 16 * ceil(H / 16)
    uint4* out;             // 2 x uint4 per pixel
    uint32_t* leaf_nid;     // per pixel, for the leaf-light shadow mask
    uint32_t item0;         // first work item (8x4-pixel tile order) of this launch

    __device__ __forceinline__ bool load(const SceneView&, uint32_t i, TravState& st) const {
        uint32_t px, py;
        if (!tile_pixel(item0 + i, pd.frameSize[0], pd.frameSize[1], px, py) || py == 0u) return false;
        st.slot = py * pd.frameSize[0] + px;
        camera_ray(pd, px, ngy16 - py, st.r.dx, st.r.dy, st.r.dz);
        st.r.ox = pd.cameraPos[0]; st.r.oy = pd.cameraPos[1]; st.r.oz = pd.cameraPos[2];
        st.t = kTMax;
        st.any = false;
        st.dup_ok = false;   // the hit leaf's light list feeds the shadow rays
        return true;
    }
    __device__ __forceinline__ void store(const SceneView&, uint32_t, const TravState& st, float) const {
        const uint32_t pix = st.slot;
        out[2u * pix] = make_uint4(st.rec0, st.rec1, st.rec2, __float_as_uint(st.t));
        out[2u * pix + 1u] = make_uint4(0u, 0u, 0u, 0u);
        leaf_nid[pix] = st.hit ? st.nid : 0xFFFFFFFFu;
    }
    __device__ __forceinline__ void skip(uint32_t i) const {
        uint32_t px, py;
        if (!tile_pixel(item0 + i, pd.frameSize[0], pd.frameSize[1], px, py)) return;
        const uint32_t pix = py * pd.frameSize[0] + px;
        out[2u * pix] = make_uint4(0u, 0u, 0u, 0u);
        out[2u * pix + 1u] = make_uint4(0u, 0u, 0u, 0u);
        leaf_nid[pix] = 0xFFFFFFFFu;
    }
    __device__ __forceinline__ bool wants_nid(const TravState&) const { return true; }
    __device__ __forceinline__ bool wants_bary(const TravState&) const { return false; }
};

// Secondary rays queued by band and kind (QueueBands). Segment e of the work items
// starts at prefix[e], prefix[n * kNumKinds] being their total. The segments run band
// by band, or -- closest_last: the two kinds of rays are traced by launches of their
// own -- the bands' any-hit kinds first and their bounce rays after them, of which a
// launch traces segments [seg0, seg1). ray.flags: bit 0 any-hit, bits 8..15 the mask
// bit, bits 16..17 the output (0 shadow mask, 1 probe mask, 2 bounce record).
// With done / flags (a pipelined camera trace), finished rays are counted per
// band and flags[b] is set once all of band b's rays are stored.
__device__ __forceinline__ void segment_of(uint32_t e, uint32_t nb, bool closest_last, uint32_t& band, uint32_t& kind) {
    if (!closest_last) {
        band = e / kNumKinds;
        kind = e - band * kNumKinds;
    } else if (e < nb * kKindBounce) {
        band = e / kKindBounce;
        kind = e - band * kKindBounce;
    } else {
        band = e - nb * kKindBounce;
        kind = kKindBounce;
    }
}

struct SecondaryPolicy {
    static constexpr bool kFinishes = true;
    const tim_rt_ray* rays;
    const uint32_t* pixel;
    const uint32_t* prefix;
    QueueBands qb;
    uint32_t* out_words;    // tracingData as u32 words (8 per pixel)
    uint4* bounce_out;
    uint32_t* done;         // finished rays per band, or null
    const uint32_t* band_total;
    volatile uint32_t* flags;
    uint32_t seg0, seg1;
    bool closest_last;

    // Work items of the launch: those of its segments.
    __device__ __forceinline__ uint32_t items() const { return __ldg(prefix + seg1) - __ldg(prefix + seg0); }
    __device__ __forceinline__ bool load(const SceneView&, uint32_t i, TravState& st) const {
        i += __ldg(prefix + seg0);
        uint32_t lo = seg0, hi = seg1;   // largest segment e with prefix[e] <= i
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(prefix + mid) <= i) lo = mid;
            else hi = mid;
        }
        uint32_t band, kind;
        segment_of(lo, qb.n, closest_last, band, kind);
        const uint32_t slot = qb.base[band] + kind * qb.cap[band] + (i - __ldg(prefix + lo));
        st.slot = slot;
        const float4* rp = reinterpret_cast<const float4*>(rays + slot);
        const float4 a = __ldg(rp), b = __ldg(rp + 1);
        st.r.ox = a.x; st.r.oy = a.y; st.r.oz = a.z;
        st.r.dx = b.x; st.r.dy = b.y; st.r.dz = b.z;
        st.t = a.w;
        st.any = (__float_as_uint(b.w) & 1u) != 0u;
        st.dup_ok = true;   // bounce rays store the hit record only
        st.slot2 = __ldg(pixel + slot);   // read now, used when the ray is stored
        return true;
    }
    // Called by all 32 lanes after a round of stores (`stored`: this lane stored
    // a ray of pixel `pix`): one count per band and warp, after each
    // storing lane's release fence; the count that completes a band follows every
    // other count of the band in the counter's order, and raises the band's flag
    // after a system-scope fence.
    __device__ __forceinline__ void finished(bool stored, uint32_t pix) const {
        if (!done) return;
        uint32_t band = 0xFFFFFFFFu;
        if (stored) {
            band = 0;
            for (uint32_t k = 1; k < qb.n; ++k) band += pix >= qb.base[k] / kNumKinds ? 1u : 0u;   // base = kNumKinds * W * row
            asm volatile("fence.acq_rel.gpu;" ::: "memory");   // this lane's stores before the warp's count
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, band);
        __syncwarp();
        const uint32_t lane = threadIdx.x & 31u;
        if (stored && lane == (uint32_t)(__ffs(peers) - 1)) {
            const uint32_t cnt = (uint32_t)__popc(peers);
            if (atomicAdd(done + band, cnt) + cnt == __ldg(band_total + band)) {
                __threadfence_system();
                flags[band] = 1u;
            }
        }
    }
    __device__ __forceinline__ void store(const SceneView&, uint32_t, const TravState& st, float) const {
        const uint32_t p = st.slot2;
        if (!st.any) {   // a bounce ray
            bounce_out[p] = make_uint4(st.rec0, st.rec1, st.rec2, __float_as_uint(st.t));
        } else if (st.hit) {
            const uint32_t fl = __float_as_uint(__ldg(reinterpret_cast<const float*>(rays + st.slot) + 7));
            const uint32_t kind = (fl >> 16) & 3u, bit = (fl >> 8) & 0xFFu;
            atomicOr(out_words + 8u * p + 4u + kind, 1u << bit);
        }
    }
    __device__ __forceinline__ void skip(uint32_t) const {}
    __device__ __forceinline__ bool wants_nid(const TravState&) const { return false; }
    __device__ __forceinline__ bool wants_bary(const TravState&) const { return false; }
};

// -------------------------------------------------------------------- persistent loop

// sdepth: traversal-stack entries per thread (the tree depth; <= 32). The stack
// lives in dynamic shared memory, entry k of thread t at [k * BLOCK + t].
template <int BLOCK, bool WIDE, bool STATS, class Policy>
__global__ void __launch_bounds__(BLOCK, WIDE ? 896 / BLOCK : 1024 / BLOCK) k_persistent(SceneView s, Policy P, uint32_t n_static,
                                                      uint32_t* counter, uint32_t* err,
                                                      unsigned long long* stats, int sdepth, int knobs) {
    extern __shared__ uint32_t stack_mem[];
    // knobs: refill threshold (bits 0..7), phase-switch threshold (bits 8..15)
    const int refill_min = knobs & 0xFF;
    const uint32_t phase_sw = (uint32_t)(knobs >> 8) & 0xFFu;
    uint32_t* stk = stack_mem + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n = items_of(P, n_static);
    const uint32_t root = s.num_nodes == 1u ? kNidLeafBit : 0u;   // baseRaytracingPass.glsl:20

    TravState st;
    st.done = true;
    // active: a ray is being traversed; pending: its traversal ended and its
    // result waits to be finished (8-wide proof) and stored. Pending lanes are
    // finished together when the warp refills, so that end-of-ray work runs
    // converged instead of once per lane as lanes end at different steps.
    bool active = false, pending = false, exhausted = false;
    uint32_t idx = 0;
    auto start = [&](uint32_t item) {
        idx = item;
        if (P.load(s, idx, st)) {
            st.t0 = st.t;
            st.err = err;
            if (WIDE) wide_init(s, st, stk);
            else trav_init(st, root);
            active = true;
        } else {
            P.skip(idx);
        }
    };
    for (;;) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !active);
        // refill once at least refill_min lanes are idle (32: whole-warp
        // batches, which keeps coherent rays of a batch in lockstep); after the
        // last ray was handed out, finish pending lanes as they come
        if (idle && (exhausted || __popc(idle) >= refill_min || idle == 0xFFFFFFFFu)) {
            const bool stored = pending;
            if (pending) {
                pending = false;
                if (WIDE) wide_finish_or_walk(s, st, err);
                P.store(s, idx, st, st.t0);
                if (STATS) {
                    atomicAdd(stats + 0, 1ull);
                    atomicAdd(stats + 1, (unsigned long long)st.c_node);
                    atomicAdd(stats + 2, (unsigned long long)st.c_leaf);
                    atomicAdd(stats + 3, (unsigned long long)st.c_tri);
                    atomicAdd(stats + 4, (unsigned long long)st.c_reload);
                }
            }
            if constexpr (finishes<Policy>::value) P.finished(stored, st.slot2);
            if (!exhausted) {
                const int leader = __ffs(idle) - 1;
                uint32_t base = 0;
                if ((int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(idle));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if ((uint64_t)base + (uint32_t)__popc(idle) >= n) exhausted = true;
                if (!active) {
                    const uint32_t my = base + __popc(idle & lanemask_lt());
                    if (my < n) start(my);
                }
            }
        }
        if (__ballot_sync(0xFFFFFFFFu, active || pending) == 0u) {
            if (exhausted) break;
            continue;
        }
        if (WIDE) {
            wide_step_warp<BLOCK>(s, st, active, stk, err, sdepth, phase_sw);   // all lanes: warp-synchronous step
        } else {
            plain_step_warp<BLOCK, leaf_kind<Policy>::value>(s, st, active, stk, err, sdepth, phase_sw);
        }
        if (active && st.done) {
            active = false;
            pending = true;
        }
    }
}

// -------------------------------------------------------------------- secondary ray generation

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}
__device__ __forceinline__ float u01(uint32_t h) { return (float)(h >> 8) * (1.0f / 16777216.0f); }

// Cosine-weighted direction about unit normal (nx,ny,nz): Malley's method with
// a rejection-sampled disk point and the orthonormal basis of Duff et al.,
// "Building an Orthonormal Basis, Revisited" (JCGT 2017).
__device__ __forceinline__ void bounce_dir(float nx, float ny, float nz, uint32_t pixel, uint32_t seed, float& dx,
                                           float& dy, float& dz) {
    float x = 0.f, y = 0.f;
    for (uint32_t k = 0; k < 16u; ++k) {
        const uint32_t h0 = hash32(pixel * 2u + 0x9E3779B9u * (seed + 1u) + k * 0x85EBCA6Bu);
        const uint32_t h1 = hash32(h0 ^ 0x27D4EB2Fu);
        const float a = u01(h0) * 2.0f - 1.0f, b = u01(h1) * 2.0f - 1.0f;
        if (a * a + b * b < 1.0f) { x = a; y = b; break; }
    }
    const float z = sqrtf(fmaxf(0.0f, 1.0f - x * x - y * y));
    const float sign = copysignf(1.0f, nz);
    const float a = -1.0f / (sign + nz);
    const float b = nx * ny * a;
    const float b1x = 1.0f + sign * nx * nx * a, b1y = sign * b, b1z = -sign * nx;
    const float b2x = b, b2y = sign + ny * ny * a, b2z = -ny;
    dx = (b1x * x + b2x * y) + nx * z;
    dy = (b1y * x + b2y * y) + ny * z;
    dz = (b1z * x + b2z * y) + nz * z;
}

struct GenParams {
    tim_rt_pass_data pd;
    uint32_t flags;
    uint32_t seed;
    uint32_t ngy16;
    uint32_t tiles_x;
    const uint32_t* tile_counts;
    const uint32_t* tile_lists;
    uint32_t* out_words;
    const uint32_t* leaf_nid;
    uint4* bounce_out;
    tim_rt_ray* q_rays;
    uint32_t* q_pixel;
    uint32_t* q_counts;     // counters [band][kind]
    uint32_t* prefix;       // first work item per segment, then their total
    uint32_t* band_total;
    uint32_t* ticket;       // blocks done
    volatile uint32_t* flags_host;   // per band, or null
    bool closest_last;      // see SecondaryPolicy
    QueueBands qb;
    uint32_t item0, item1;  // work items (8x4-pixel tile order) of this launch
};

__device__ __forceinline__ void lpf_position(const tim_rt_pass_data& pd, uint32_t cx, uint32_t cy, uint32_t cz,
                                             float& x, float& y, float& z) {
    // lightprobHelpers.glsl:63-69 getLightProbPosition
    const float stx = (pd.sceneMaxExtent[0] - pd.sceneMinExtent[0]) / (float)pd.lpfResolution[0];
    const float sty = (pd.sceneMaxExtent[1] - pd.sceneMinExtent[1]) / (float)pd.lpfResolution[1];
    const float stz = (pd.sceneMaxExtent[2] - pd.sceneMinExtent[2]) / (float)pd.lpfResolution[2];
    x = pd.sceneMinExtent[0] + stx * ((float)cx + 0.5f);
    y = pd.sceneMinExtent[1] + sty * ((float)cy + 0.5f);
    z = pd.sceneMinExtent[2] + stz * ((float)cz + 0.5f);
}

// A warp's places in the queue: lane k holds the lanes that append a ray of kind k and,
// after reserve(), the first of their slots of that kind in the warp's band (uniform
// across the warp). All kinds' counters are bumped by one atomic instruction, one kind a
// lane: kind by kind, each with the round trip to the L2 before its stores, the 26 kinds
// bound the generators (0.17 -> 0.11 ms for the 1080p frame with tile lights and bounces,
// 0.17 -> 0.08 for 1279x719 with probe visibility, 0.23 -> 0.11 for 2.1M probe rays).
struct Places {
    uint32_t mask = 0, base = 0;
    // every lane calls; `has`: this lane appends a ray of `kind`
    __device__ __forceinline__ void want(uint32_t kind, bool has) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, has);
        if ((threadIdx.x & 31u) == kind) mask = m;
    }
    __device__ __forceinline__ void reserve(const GenParams& g, uint32_t band) {
        const uint32_t lane = threadIdx.x & 31u;
        if (lane < kNumKinds && mask) base = atomicAdd(g.q_counts + band * kNumKinds + lane, (uint32_t)__popc(mask));
    }
    // Writes this lane's ray of `kind`, lane order preserved inside the segment; every
    // lane calls, with the `has` of want().
    __device__ __forceinline__ void put(const GenParams& g, uint32_t band, uint32_t kind, bool has, uint32_t pix,
                                        float ox, float oy, float oz, float tmax, float dx, float dy, float dz,
                                        uint32_t flags) const {
        const uint32_t m = __shfl_sync(0xFFFFFFFFu, mask, kind), b = __shfl_sync(0xFFFFFFFFu, base, kind);
        if (!has) return;
        const uint32_t off = b + __popc(m & lanemask_lt()), cap = g.qb.cap[band];
        if (off < cap) {
            const uint64_t slot = (uint64_t)g.qb.base[band] + (uint64_t)kind * cap + off;
            float4* rp = reinterpret_cast<float4*>(g.q_rays + slot);
            rp[0] = make_float4(ox, oy, oz, tmax);
            rp[1] = make_float4(dx, dy, dz, __uint_as_float(flags));
            g.q_pixel[slot] = pix;
        }
    }
};

// One light of a hit's list, seen from (hx, hy, hz) (evalShadow, bvhLighting.glsl:114-134:
// sphere lights only): its mask bit, whether it is in range, the distance, and where.
struct LightRay {
    uint32_t bit;
    bool sphere, in_range;
    float dist, x, y, z;
};
__device__ __forceinline__ LightRay light_ray(const SceneView& s, uint32_t li, float hx, float hy, float hz) {
    LightRay l{li + 1u, false, false, 1.f, 0.f, 0.f, 0.f};
    const float* L = s.lights + 14u * li;
    if (__float_as_uint(__ldg(L)) == kLightSphere && l.bit < 32u) {
        l.sphere = true;
        l.x = __ldg(L + 1) - hx;
        l.y = __ldg(L + 2) - hy;
        l.z = __ldg(L + 3) - hz;
        l.dist = sqrtf(dot3(l.x, l.y, l.z, l.x, l.y, l.z));
        l.in_range = l.dist < __ldg(L + 4);
    }
    return l;
}

// The light list of leaf `nid`, and its length.
__device__ __forceinline__ const uint32_t* leaf_lights(const SceneView& s, uint32_t nid, uint32_t& count) {
    const uint32_t off = __ldg(reinterpret_cast<const uint32_t*>(s.nodes + 4u * nid) + 3);
    const uint32_t hdr = leaf_header(s, off);
    uint32_t skip = 3u * (hdr & ((1u << kTriBits) - 1u));
    skip += (hdr >> kTriBits) & ((1u << kBlasBits) - 1u);
    skip += (hdr >> (kTriBits + kBlasBits)) & ((1u << kPrimBits) - 1u);
    count = (hdr >> (kTriBits + kBlasBits + kPrimBits)) & ((1u << kLightBits) - 1u);
    return s.leaf + skip + 1u + off;
}

// The shadow rays to a list of lights, counted (before reserve()): lights out of range set
// their bit directly (evalShadow returns true, bvhLighting.glsl:121-124). Lights past every
// lane's count emit nothing: the loop ends at the warp's largest count.
__device__ __forceinline__ uint32_t want_lights(const SceneView& s, Places& pl, const uint32_t* list, uint32_t count,
                                                uint32_t jmax, float hx, float hy, float hz) {
    uint32_t direct_bits = 0;
    for (uint32_t j = 0; j < jmax; ++j) {
        bool has = false;
        if (j < count) {
            const LightRay l = light_ray(s, __ldg(list + j), hx, hy, hz);
            has = l.sphere && l.in_range;
            if (l.sphere && !l.in_range) direct_bits |= 1u << l.bit;
        }
        pl.want(kKindLight0 + j, has);
    }
    return direct_bits;
}

// The same rays, written: each lane those that want_lights() found, a light that no lane
// of the warp reaches not looked at again (1080p frame 0.116 -> 0.108 ms, without bounces
// 0.095 -> 0.085; 2.1M probe rays 0.120 -> 0.101).
__device__ __forceinline__ void put_lights(const SceneView& s, const GenParams& g, const Places& pl, uint32_t band,
                                           const uint32_t* list, uint32_t jmax, uint32_t pix, float hx, float hy, float hz) {
    for (uint32_t j = 0; j < jmax; ++j) {
        const uint32_t lanes = __shfl_sync(0xFFFFFFFFu, pl.mask, kKindLight0 + j);
        if (!lanes) continue;
        const bool has = lanes >> (threadIdx.x & 31u) & 1u;
        float dx = 0.f, dy = 0.f, dz = 0.f, dist = 1.f;
        uint32_t bit = 0;
        if (has) {
            const LightRay l = light_ray(s, __ldg(list + j), hx, hy, hz);
            bit = l.bit;
            dist = l.dist;
            dx = l.x / dist;
            dy = l.y / dist;
            dz = l.z / dist;
        }
        pl.put(g, band, kKindLight0 + j, has, pix, hx, hy, hz, dist, dx, dy, dz, 1u | (bit << 8));
    }
}

// Ends a generator: the last block to finish turns the segment counts into each segment's
// first work item (prefix[e], see SecondaryPolicy, the counts clamped to the capacities)
// and the rays per band. A band without secondary rays is final already: its flag (when
// there are flags) is raised here.
__device__ __forceinline__ void finish_queue(const GenParams& g) {
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0u) {
        __threadfence();
        last = atomicAdd(g.ticket, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32u) return;
    __threadfence();
    const uint32_t lane = threadIdx.x, nb = g.qb.n, n = nb * kNumKinds;
    uint32_t acc = 0;
    for (uint32_t e0 = 0; e0 < n; e0 += 32u) {
        const uint32_t e = e0 + lane;
        uint32_t c = 0;
        if (e < n) {
            uint32_t band, kind;
            segment_of(e, nb, g.closest_last, band, kind);
            c = min(__ldcg(g.q_counts + band * kNumKinds + kind), g.qb.cap[band]);
        }
        uint32_t sum = c;
#pragma unroll
        for (uint32_t k = 1; k < 32u; k <<= 1) {
            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, sum, k);
            if (lane >= k) sum += v;
        }
        if (e < n) g.prefix[e] = acc + sum - c;
        acc += __shfl_sync(0xFFFFFFFFu, sum, 31);
    }
    if (lane == 0u) g.prefix[n] = acc;
    if (lane < nb) {
        uint32_t t = 0;
        for (uint32_t k = 0; k < kNumKinds; ++k) t += min(__ldcg(g.q_counts + lane * kNumKinds + k), g.qb.cap[lane]);
        g.band_total[lane] = t;
        if (g.flags_host && t == 0u) {
            __threadfence_system();
            g.flags_host[lane] = 1u;
        }
    }
}

// For each camera hit, queue the rays of computeAdditionalHitData
// (baseRaytracingPass.glsl:85-97): the sun shadow ray and one ray per light of
// the hit leaf's list (bvhLighting.glsl:143-163) or of the pixel's tile list,
// the 8 probe-visibility segments (bvhLighting.glsl:165-184) and the bounce.
// One thread per pixel, pixels in 8x4 tiles.
__global__ void __launch_bounds__(256) k_gen_secondary(SceneView s, GenParams g) {
    const tim_rt_pass_data& pd = g.pd;
    const uint32_t W = pd.frameSize[0], H = pd.frameSize[1];
    const uint32_t i = g.item0 + blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t px = 0, py = 0;
    const bool valid = i < g.item1 && tile_pixel(i, W, H, px, py);
    const uint32_t pix = py * W + px;
    // the warp's band: all its pixels lie in one 8x4 tile, bands end on tile rows
    const uint32_t band = band_of_row(g.qb, (i >> 5) / ((W + 7u) >> 3) * 4u);
    uint4 rec = make_uint4(0, 0, 0, 0);
    if (valid) rec = reinterpret_cast<const uint4*>(g.out_words)[2u * pix];
    const float t = __uint_as_float(rec.w);
    const bool hit = valid && py != 0u && t < kTMax;
    const uint32_t gx = px, gy = g.ngy16 - py;
    float dx = 0.f, dy = 0.f, dz = 0.f, hx = 0.f, hy = 0.f, hz = 0.f;
    if (hit) {
        camera_ray(pd, gx, gy, dx, dy, dz);
        // baseRaytracingPass.glsl:91 hitPos = from + dir * t
        hx = pd.cameraPos[0] + dx * t;
        hy = pd.cameraPos[1] + dy * t;
        hz = pd.cameraPos[2] + dz * t;
    }
    // light list of the tile or of the hit leaf
    const uint32_t* list = nullptr;
    uint32_t count = 0;
    if (hit) {
        if (g.flags & TIM_RT_CAM_TILE_LIGHTS) {
            const uint32_t tile = (gy / 16u) * g.tiles_x + gx / 16u;
            list = g.tile_lists + 16u * tile;
            count = min(g.tile_counts[tile], 16u);
        } else {
            list = leaf_lights(s, g.leaf_nid[pix], count);
        }
    }
    const uint32_t jmax = __reduce_max_sync(0xFFFFFFFFu, count);   // usually uniform: one tile's list
    Places pl;
    pl.want(kKindSun, hit);
    const uint32_t direct_bits = want_lights(s, pl, list, count, jmax, hx, hy, hz);
    if (g.flags & TIM_RT_CAM_PROB_MASK)
        for (uint32_t k = 0; k < 8u; ++k) pl.want(kKindProbe0 + k, hit);
    if (g.flags & TIM_RT_CAM_BOUNCE) pl.want(kKindBounce, hit);
    pl.reserve(g, band);
    // sun ray, tmax = TMAX (bvhLighting.glsl:148-149)
    pl.put(g, band, kKindSun, hit, pix, hx, hy, hz, kTMax, -pd.sunDir[0], -pd.sunDir[1], -pd.sunDir[2], 1u);
    put_lights(s, g, pl, band, list, jmax, pix, hx, hy, hz);
    if (g.flags & TIM_RT_CAM_PROB_MASK) {
        // lightprobHelpers.glsl:71-77 getLightProbCoordUVW and bvhLighting.glsl:170-180
        uint32_t cx = 0, cy = 0, cz = 0;
        if (hit) {
            const uint32_t* res = pd.lpfResolution;
            const float stx = (pd.sceneMaxExtent[0] - pd.sceneMinExtent[0]) / (float)res[0];
            const float sty = (pd.sceneMaxExtent[1] - pd.sceneMinExtent[1]) / (float)res[1];
            const float stz = (pd.sceneMaxExtent[2] - pd.sceneMinExtent[2]) / (float)res[2];
            float ux = (hx - pd.sceneMinExtent[0]) / stx - 0.5f;
            float uy = (hy - pd.sceneMinExtent[1]) / sty - 0.5f;
            float uz = (hz - pd.sceneMinExtent[2]) / stz - 0.5f;
            ux = fminf(fmaxf(ux, 0.0f), (float)res[0] - 1.0f);
            uy = fminf(fmaxf(uy, 0.0f), (float)res[1] - 1.0f);
            uz = fminf(fmaxf(uz, 0.0f), (float)res[2] - 1.0f);
            const uint32_t ix = (uint32_t)(int32_t)ux, iy = (uint32_t)(int32_t)uy, iz = (uint32_t)(int32_t)uz;
            cx = min(ix, res[0] - 2u);
            cy = min(iy, res[1] - 2u);
            cz = min(iz, res[2] - 2u);
        }
        for (uint32_t k = 0; k < 8u; ++k) {
            float qx = 0.f, qy = 0.f, qz = 0.f;
            if (hit) lpf_position(pd, cx + (k & 1u), cy + ((k >> 1) & 1u), cz + ((k >> 2) & 1u), qx, qy, qz);
            pl.put(g, band, kKindProbe0 + k, hit, pix, hx, hy, hz, 1.0f, qx - hx, qy - hy, qz - hz,
                   1u | (k << 8) | (1u << 16));
        }
    }
    if (g.flags & TIM_RT_CAM_BOUNCE) {
        float bx = 0.f, by = 0.f, bz = 0.f;
        if (hit) {
            // geometric normal of the hit triangle, facing the incoming ray
            const uint32_t i0 = rec.x + (rec.y & 0xFFFFu), i1 = rec.x + (rec.y >> 16), i2 = rec.x + (rec.z & 0xFFFFu);
            const float p0x = s.pos[3u * i0], p0y = s.pos[3u * i0 + 1], p0z = s.pos[3u * i0 + 2];
            const float e1x = s.pos[3u * i1] - p0x, e1y = s.pos[3u * i1 + 1] - p0y, e1z = s.pos[3u * i1 + 2] - p0z;
            const float e2x = s.pos[3u * i2] - p0x, e2y = s.pos[3u * i2 + 1] - p0y, e2z = s.pos[3u * i2 + 2] - p0z;
            float nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
            const float nl = sqrtf(dot3(nx, ny, nz, nx, ny, nz));
            nx = nx / nl; ny = ny / nl; nz = nz / nl;
            if (dot3(nx, ny, nz, dx, dy, dz) > 0.0f) { nx = -nx; ny = -ny; nz = -nz; }
            bounce_dir(nx, ny, nz, pix, g.seed, bx, by, bz);
        }
        pl.put(g, band, kKindBounce, hit, pix, hx, hy, hz, kTMax, bx, by, bz, 2u << 16);
    }
    if (valid) {
        g.out_words[8u * pix + 4u] = direct_bits;
        g.out_words[8u * pix + 5u] = 0u;
        if (g.bounce_out) g.bounce_out[pix] = make_uint4(0u, 0u, 0u, 0u);
    }
    finish_queue(g);
}

// Adds the frame's ray count (primary rays of rows 1..H-1 plus the secondary queue).
__global__ void k_add_ray_count(uint64_t* dst, uint64_t primary, const uint32_t* total) {
    *dst += primary + *total;
}

// -------------------------------------------------------------------- tile light culling

// cullFrustum.glsl:9-13 computePlan
__device__ __forceinline__ void compute_plan(float p1x, float p1y, float p1z, float p2x, float p2y, float p2z,
                                             float p3x, float p3y, float p3z, float4& pl) {
    const float ax = p1x - p2x, ay = p1y - p2y, az = p1z - p2z;
    const float bx = p3x - p2x, by = p3y - p2y, bz = p3z - p2z;
    float nx = ay * bz - az * by, ny = az * bx - ax * bz, nz = ax * by - ay * bx;
    const float l = sqrtf(dot3(nx, ny, nz, nx, ny, nz));
    nx = nx / l; ny = ny / l; nz = nz / l;
    pl = make_float4(nx, ny, nz, -dot3(nx, ny, nz, p2x, p2y, p2z));
}

// One warp per tile: lanes test lights lane, lane+32, ...; survivors are
// compacted with a ballot in ascending light order (cullFrustum.glsl:63-100,136-151,
// collision.glsl:219-227).
__global__ void __launch_bounds__(256) k_cull_lights(SceneView s, tim_rt_pass_data pd, uint32_t tiles_x,
                                                     uint32_t tiles_y, uint32_t* counts, uint32_t* lists) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    if (warp >= tiles_x * tiles_y) return;
    const uint32_t wx = warp % tiles_x, wy = warp / tiles_x;
    const float* c00 = pd.frustumCorner00;
    const float* c10 = pd.frustumCorner10;
    const float* c01 = pd.frustumCorner01;
    const float sxx = (c10[0] - c00[0]) / (float)tiles_x, sxy = (c10[1] - c00[1]) / (float)tiles_x,
                sxz = (c10[2] - c00[2]) / (float)tiles_x;
    const float syx = (c01[0] - c00[0]) / (float)tiles_y, syy = (c01[1] - c00[1]) / (float)tiles_y,
                syz = (c01[2] - c00[2]) / (float)tiles_y;
    const float fx0 = (float)wx, fx1 = (float)(wx + 1u), fy0 = (float)wy, fy1 = (float)(wy + 1u);
    float blx = (c00[0] + sxx * fx0) + syx * fy0, bly = (c00[1] + sxy * fx0) + syy * fy0, blz = (c00[2] + sxz * fx0) + syz * fy0;
    float brx = (c00[0] + sxx * fx1) + syx * fy0, bry = (c00[1] + sxy * fx1) + syy * fy0, brz = (c00[2] + sxz * fx1) + syz * fy0;
    float tlx = (c00[0] + sxx * fx0) + syx * fy1, tly = (c00[1] + sxy * fx0) + syy * fy1, tlz = (c00[2] + sxz * fx0) + syz * fy1;
    float trx = (c00[0] + sxx * fx1) + syx * fy1, try_ = (c00[1] + sxy * fx1) + syy * fy1, trz = (c00[2] + sxz * fx1) + syz * fy1;
    const float dxx = sxx * 0.25f, dxy = sxy * 0.25f, dxz = sxz * 0.25f;
    const float dyx = syx * 0.25f, dyy = syy * 0.25f, dyz = syz * 0.25f;
    blx = (blx - dxx) - dyx; bly = (bly - dxy) - dyy; blz = (blz - dxz) - dyz;
    brx = (brx + dxx) - dyx; bry = (bry + dxy) - dyy; brz = (brz + dxz) - dyz;
    tlx = (tlx - dxx) + dyx; tly = (tly - dxy) + dyy; tlz = (tlz - dxz) + dyz;
    trx = (trx + dxx) + dyx; try_ = (try_ + dxy) + dyy; trz = (trz + dxz) + dyz;
    const float cx = pd.cameraPos[0], cy = pd.cameraPos[1], cz = pd.cameraPos[2];
    float4 pl[4];
    compute_plan(cx, cy, cz, tlx, tly, tlz, blx, bly, blz, pl[0]);
    compute_plan(cx, cy, cz, brx, bry, brz, trx, try_, trz, pl[1]);
    compute_plan(cx, cy, cz, trx, try_, trz, tlx, tly, tlz, pl[2]);
    compute_plan(cx, cy, cz, blx, bly, blz, brx, bry, brz, pl[3]);
    uint32_t cnt = 0;
    uint32_t* lst = lists + 16u * warp;
    for (uint32_t base = 0; base < s.num_lights && cnt < 16u; base += 32u) {
        const uint32_t i = base + lane;
        bool inside = false;
        if (i < s.num_lights) {
            const float* L = s.lights + 14u * i;
            const float px = __ldg(L + 1), py = __ldg(L + 2), pz = __ldg(L + 3), r = __ldg(L + 4);
            inside = true;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (dot3(pl[k].x, pl[k].y, pl[k].z, px, py, pz) + pl[k].w < -r) inside = false;
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, inside);
        const uint32_t pos = cnt + __popc(m & lanemask_lt());
        if (inside && pos < 16u) lst[pos] = i;
        cnt += __popc(m);
    }
    cnt = min(cnt, 16u);
    if (lane >= cnt && lane < 16u) lst[lane] = 0xFFFFFFFFu;
    if (lane == 0) counts[warp] = cnt;
}

// -------------------------------------------------------------------- launchers

template <int BLOCK, bool WIDE, bool STATS, class Policy>
static void launch_block(const SceneView& s, const Policy& P, uint32_t n_static,
                         uint32_t* counter, uint32_t* err, unsigned long long* stats, int depth, int refill,
                         cudaStream_t stream) {
    static GridCache cache;
    const int grid = grid_of<BLOCK, Policy>(cache, k_persistent<BLOCK, WIDE, STATS, Policy>, depth, kStackSize);
    k_persistent<BLOCK, WIDE, STATS, Policy><<<grid, BLOCK, stack_bytes<BLOCK, Policy>(depth), stream>>>(
        s, P, n_static, counter, err, stats, depth, refill);
}

template <bool WIDE, class Policy>
static cudaError_t launch_persistent(const SceneView& s, const Policy& P, uint32_t n_static,
                                     uint32_t* counter, uint32_t* err, cudaStream_t stream, const LaunchConfig& cfg) {
    int depth = WIDE ? (int)s.wide_depth : (int)s.depth;
    if (cfg.stack_depth > depth) depth = cfg.stack_depth;
    depth = depth < 1 ? 1 : (depth > kStackSize ? kStackSize : depth);
    const int refill = launch_knobs(cfg);
    if (cfg.stats) {
        launch_block<128, WIDE, true>(s, P, n_static, counter, err, cfg.stats, depth, refill, stream);
        return cudaGetLastError();
    }
    switch (cfg.block) {
        case 64: launch_block<64, WIDE, false>(s, P, n_static, counter, err, nullptr, depth, refill, stream); break;
        case 256: launch_block<256, WIDE, false>(s, P, n_static, counter, err, nullptr, depth, refill, stream); break;
        default: launch_block<128, WIDE, false>(s, P, n_static, counter, err, nullptr, depth, refill, stream); break;
    }
    return cudaGetLastError();
}

static bool use_walk(const SceneView& s, const LaunchConfig& cfg) { return !cfg.stats && has_walk(s, cfg.wide); }

// The general kernel: counting launches, two-level scenes, scenes without the trees of the
// walks.
template <class Policy>
static cudaError_t launch_general(const SceneView& s, const Policy& P, uint32_t n, uint32_t* counter, uint32_t* err,
                                  cudaStream_t stream, const LaunchConfig& cfg) {
    return cfg.wide ? launch_persistent<true>(s, P, n, counter, err, stream, cfg)
                    : launch_persistent<false>(s, P, n, counter, err, stream, cfg);
}

cudaError_t launch_trace_batch(const SceneView& s, const tim_rt_ray* rays, uint32_t n, uint32_t mode, uint32_t* hit,
                               uint32_t* nid, float* bary, uint32_t* counter, uint32_t* err, cudaStream_t stream,
                               const LaunchConfig& cfg) {
    BatchPolicy P{rays, reinterpret_cast<uint4*>(hit), nid, reinterpret_cast<float2*>(bary), mode & 0xFFu};
    if (mode & TIM_RT_TRACE_TLAS) {   // any-hit only, binary form only (checked by the callers)
        TlasBatchPolicy T;
        static_cast<BatchPolicy&>(T) = P;
        return launch_persistent<false>(s, T, n, counter, err, stream, cfg);
    }
    if (!use_walk(s, cfg)) return launch_general(s, P, n, counter, err, stream, cfg);
    if (P.mode == TIM_RT_MODE_CLOSEST) return launch_rays<false>(s, P, n, counter, err, stream, cfg);
    if (P.mode == TIM_RT_MODE_ANY) return launch_rays<true>(s, P, n, counter, err, stream, cfg);
    KindBatchPolicy K;
    static_cast<BatchPolicy&>(K) = P;
    K.kind = 0u;
    const cudaError_t e = launch_rays<false>(s, K, n, counter, err, stream, cfg, kPairFirst);
    if (e != cudaSuccess) return e;
    K.kind = TIM_RT_RAY_ANY;
    return launch_rays<true>(s, K, n, counter + 1, err, stream, cfg, kPairSecond);
}

// The queue's counters (laid out as kernels.h says) as a generator and its launch use them.
static void queue_counters(uint32_t* counters, const QueueBands& qb, volatile uint32_t* flags, bool closest_last,
                           GenParams& g) {
    g.qb = qb;
    g.q_counts = counters + 2;
    g.prefix = counters + 2u + kNumKinds * qb.n;
    g.band_total = g.prefix + kNumKinds * qb.n + 1u + qb.n;
    g.ticket = counters + 4u + 54u * qb.n;
    g.flags_host = flags;
    g.closest_last = closest_last;
}

// Traces the queue a generator with these counters left: the rays in one launch, or, where
// the scene has_walk, the any-hit rays and the bounce rays in launches of their own: in the
// binary form they walk different trees, of which a warp of both kinds would walk each with
// part of its lanes, and in both forms an any-hit ray carries half the state.
static cudaError_t launch_secondary(const SceneView& s, const GenParams& g, uint32_t* counters, uint32_t* err,
                                    cudaStream_t stream, const LaunchConfig& cfg, bool bounces) {
    const uint32_t nb = g.qb.n;
    SecondaryPolicy P{};
    P.rays = g.q_rays;
    P.pixel = g.q_pixel;
    P.prefix = g.prefix;
    P.qb = g.qb;
    P.out_words = g.out_words;
    P.bounce_out = g.bounce_out;
    P.flags = g.flags_host;
    P.done = P.flags ? g.prefix + kNumKinds * nb + 1u : nullptr;
    P.band_total = g.band_total;
    P.closest_last = g.closest_last;
    P.seg0 = 0u;
    P.seg1 = nb * kNumKinds;
    if (!g.closest_last) return launch_general(s, P, 0u, counters + 1, err, stream, cfg);
    if (bounces) {
        P.seg0 = nb * kKindBounce;
        // with bands both launches must get on together, as a band is final after both:
        // half of the GPU for the bounce rays (the 1080p frame through host buffers takes
        // 2.57 ms with a half, 2.58 with a third, 2.62 with a quarter)
        const cudaError_t e = launch_rays<false>(s, P, 0u, counters + 3u + 54u * nb, err, stream, cfg, kPairFirst,
                                                 nb > 1u ? 2 : 1);
        if (e != cudaSuccess) return e;
        P.seg0 = 0u;
    }
    P.seg1 = nb * kKindBounce;
    return launch_rays<true>(s, P, 0u, counters + 1, err, stream, cfg, bounces ? kPairSecond : kAlone);
}

uint32_t camera_queue_segment(uint32_t W, uint32_t H) { return W * H; }
uint32_t camera_queue_kinds() { return kNumKinds; }
uint32_t probe_queue_kinds() { return kKindProbe0; }

cudaError_t launch_camera(const SceneView& s, const tim_rt_pass_data& pd, uint32_t flags, uint32_t seed,
                          const uint32_t* tile_counts, const uint32_t* tile_lists, uint32_t* out, uint32_t* bounce_out,
                          uint32_t* leaf_nid, tim_rt_ray* q_rays, uint32_t* q_pixel, uint32_t seg_cap,
                          uint32_t* counters, uint32_t* err, uint64_t* d_ray_count, cudaStream_t stream,
                          const LaunchConfig& cfg, uint32_t row_begin, uint32_t row_end, const CameraBands* bands) {
    const uint32_t W = pd.frameSize[0], H = pd.frameSize[1];
    // output rows [row_begin, row_end): whole rows of 8x4-pixel tiles (row_begin a multiple of 4)
    row_end = min(row_end, H);
    if (row_begin >= row_end) return cudaSuccess;
    // the queue's bands: one (the launch's rows, segments of seg_cap slots), or the
    // caller's bands of the whole frame (segments of each band's pixels)
    QueueBands qb{};
    qb.n = 1;
    qb.row[0] = row_begin;
    qb.row[1] = row_end;
    qb.cap[0] = seg_cap;
    if (bands && bands->n > 1u) {
        if (bands->n > kMaxCamBands || row_begin != 0u || row_end != H || seg_cap != W * H) return cudaErrorInvalidValue;
        qb.n = bands->n;
        for (uint32_t b = 0; b <= qb.n; ++b) qb.row[b] = bands->row[b];
        if (qb.row[0] != 0u || qb.row[qb.n] != H) return cudaErrorInvalidValue;
        for (uint32_t b = 0; b < qb.n; ++b) {
            if (qb.row[b + 1] <= qb.row[b] || qb.row[b] % 4u != 0u) return cudaErrorInvalidValue;
            qb.base[b] = kNumKinds * W * qb.row[b];
            qb.cap[b] = W * (qb.row[b + 1] - qb.row[b]);
        }
    }
    volatile uint32_t* flags_host = bands && bands->n > 1u ? bands->flags : nullptr;
    const uint32_t tiles_x = (W + 7u) >> 3;
    const uint32_t item0 = (row_begin >> 2) * tiles_x * 32u;
    const uint32_t item1 = min(tiled_work_items(W, H), ((row_end + 3u) >> 2) * tiles_x * 32u);
    const uint32_t items = item1 - item0;
    const uint32_t ngy16 = 16u * ((H + 15u) / 16u);
    // counters: [0] pixel work, [1] secondary work, then the bands' kind counts, their
    // prefix and the bands' finished rays
    CameraPolicy CP{pd, ngy16, reinterpret_cast<uint4*>(out), leaf_nid, item0};
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[0], stream);
    // primary rays: a warp refills only when all 32 lanes are idle, so it always
    // traces one whole 8x4-pixel tile together (measured fastest for these
    // coherent rays; the secondary launch keeps the configured threshold)
    LaunchConfig pcfg = cfg;
    pcfg.refill_min = 32;
    if (flags & TIM_RT_CAM_PRIMARY_BINARY) pcfg.wide = false;
    cudaError_t e = use_walk(s, pcfg) ? launch_rays<false>(s, CP, items, counters + 0, err, stream, pcfg)
                                      : launch_general(s, CP, items, counters + 0, err, stream, pcfg);
    if (e != cudaSuccess) return e;
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[1], stream);
    GenParams g;
    g.pd = pd;
    g.flags = flags;
    g.seed = seed;
    g.ngy16 = ngy16;
    g.tiles_x = (W + 15u) / 16u;
    g.tile_counts = tile_counts;
    g.tile_lists = tile_lists;
    g.out_words = out;
    g.leaf_nid = leaf_nid;
    g.bounce_out = reinterpret_cast<uint4*>(bounce_out);
    g.q_rays = q_rays;
    g.q_pixel = q_pixel;
    g.item0 = item0;
    g.item1 = item1;
    queue_counters(counters, qb, flags_host, use_walk(s, cfg), g);
    k_gen_secondary<<<(items + 255u) / 256u, 256, 0, stream>>>(s, g);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[2], stream);
    LaunchConfig cfg2 = cfg;   // the secondary kernel counts into stats[8..12]
    if (cfg.stats) cfg2.stats = cfg.stats + 8;
    e = launch_secondary(s, g, counters, err, stream, cfg2, (flags & TIM_RT_CAM_BOUNCE) != 0u);
    const uint32_t* total = counters + 2u + 2u * kNumKinds * qb.n;
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[3], stream);
    if (e != cudaSuccess || !d_ray_count) return e;
    // primary rays of the rows traced (output row 0 is never traced)
    const uint64_t primary = (uint64_t)W * (row_end - max(row_begin, 1u));
    k_add_ray_count<<<1, 1, 0, stream>>>(d_ray_count, primary, total);
    return cudaGetLastError();
}

cudaError_t launch_cull_lights(const SceneView& s, const tim_rt_pass_data& pd, uint32_t tiles_x, uint32_t tiles_y,
                               uint32_t* counts, uint32_t* lists, cudaStream_t stream) {
    const uint32_t warps = tiles_x * tiles_y;
    const uint32_t blocks = (warps * 32u + 255u) / 256u;
    k_cull_lights<<<blocks, 256, 0, stream>>>(s, pd, tiles_x, tiles_y, counts, lists);
    return cudaGetLastError();
}

// -------------------------------------------------------------------- light-probe field

// lightprobHelpers.glsl:33-61 getLightProbCoord (LP_TILE_RES = 4)
__device__ __forceinline__ void probe_coord(uint32_t index, const uint32_t* res, uint32_t& x, uint32_t& y, uint32_t& z) {
    const uint32_t trx = res[0] / 4u, try_ = res[1] / 4u;
    uint32_t tile = index / 64u;
    const uint32_t in = index % 64u;
    z = tile / (trx * try_);
    tile = tile % (trx * try_);
    y = tile / trx;
    x = tile % trx;
    x = x * 4u + in % 4u;
    y = y * 4u + (in / 4u) % 4u;
    z = z * 4u + (in / 16u) % 4u;
}

// lightprobHelpers.glsl:63-69 getLightProbPosition
__device__ __forceinline__ void probe_position(const ProbeArgs& d, uint32_t p, float& x, float& y, float& z) {
    uint32_t cx, cy, cz;
    probe_coord(p, d.res, cx, cy, cz);
    const float stx = (d.mx[0] - d.mn[0]) / (float)d.res[0];
    const float sty = (d.mx[1] - d.mn[1]) / (float)d.res[1];
    const float stz = (d.mx[2] - d.mn[2]) / (float)d.res[2];
    x = d.mn[0] + stx * ((float)cx + 0.5f);
    y = d.mn[1] + sty * ((float)cy + 0.5f);
    z = d.mn[2] + stz * ((float)cz + 0.5f);
}

// Work item i of the shadow-ray generator: probe-major (r = i % nd), so that a
// warp takes 32 consecutive directions of one probe and its shadow rays start
// close together; results are stored probe-major (sample = probe * nd + r) as
// genLightProbField.comp:47 indexes them.
__device__ __forceinline__ uint32_t probe_sample(const ProbeArgs& d, uint32_t i, uint32_t& pl, uint32_t& r) {
    r = i % d.nd;
    pl = i / d.nd;
    return pl * d.nd + r;
}

// Work item i of the probe-ray trace. It is probe-major like the generator, except for
// octahedral directions (TIM_RT_PROBE_OCTA) on the 8-wide walk and in the general kernel,
// where it is direction-major (r = i / np: a warp traces one direction from 32
// neighbouring probes).
// An update of 32x32x8 probes x 256 directions, direction-major against probe-major:
// binary walk, 1M triangles, octahedral 3.25 / 3.05 ms, stratified 2.76 / 2.63; octahedral
// on 2,000 to 300,000 triangles and 64 to 8,192 probes 1 to 17 % in favour of the latter;
// on the 8-wide walk, 300,000 triangles, 3.48 / 4.48 ms (20,000: 2.51 / 2.81; fields of 64
// to 384 probes 6 to 43 % the other way, 0.9 / 1.2 ms at most); general kernel, 1M
// triangles, 4.17 / 4.28 ms.
__device__ __forceinline__ uint32_t probe_trace_item(const ProbeArgs& d, uint32_t i, uint32_t& pl, uint32_t& r) {
    if (!d.trace_dir_major) return probe_sample(d, i, pl, r);
    r = i / d.np;
    pl = i % d.np;
    return pl * d.nd + r;
}

struct ProbePolicy {
    ProbeArgs d;
    uint4* out;          // 2 x uint4 per sample (tracingData layout)
    uint32_t* leaf_nid;

    __device__ __forceinline__ bool load(const SceneView&, uint32_t i, TravState& st) const {
        uint32_t pl, r;
        st.slot = probe_trace_item(d, i, pl, r);
        probe_position(d, d.p0 + pl, st.r.ox, st.r.oy, st.r.oz);
        const float4 dir = __ldg(d.dirs + r);
        st.r.dx = dir.x; st.r.dy = dir.y; st.r.dz = dir.z;
        st.t = kTMax;
        st.any = false;
        st.dup_ok = false;   // the hit leaf's light list feeds the shadow rays
        return true;
    }
    __device__ __forceinline__ void store(const SceneView&, uint32_t, const TravState& st, float) const {
        out[2u * st.slot] = make_uint4(st.rec0, st.rec1, st.rec2, __float_as_uint(st.t));
        out[2u * st.slot + 1u] = make_uint4(0u, 0u, 0u, 0u);
        leaf_nid[st.slot] = st.hit ? st.nid : 0xFFFFFFFFu;
    }
    __device__ __forceinline__ void skip(uint32_t) const {}
    __device__ __forceinline__ bool wants_nid(const TravState&) const { return true; }
    __device__ __forceinline__ bool wants_bary(const TravState&) const { return false; }
};

// Shadow rays of the probe hits: the sun (tmax = TMAX) and the hit leaf's lights
// (computeAdditionalHitData / computeShadowMask, baseRaytracingPass.glsl:85-97,
// bvhLighting.glsl:143-163); the probe mask stays 0 (no USE_LPF_MASK).
__global__ void __launch_bounds__(256) k_probe_gen(SceneView s, ProbeArgs d, GenParams g, const uint32_t* leaf_nid) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = i < d.np * d.nd;
    uint32_t probe = 0, r = 0, sample = 0;
    if (valid) sample = probe_sample(d, i, probe, r);
    uint4 rec = make_uint4(0, 0, 0, 0);
    if (valid) rec = reinterpret_cast<const uint4*>(g.out_words)[2u * sample];
    const float t = __uint_as_float(rec.w);
    const bool hit = valid && t < kTMax;
    float hx = 0.f, hy = 0.f, hz = 0.f;
    if (hit) {
        float ox, oy, oz;
        probe_position(d, d.p0 + probe, ox, oy, oz);
        const float4 dir = __ldg(d.dirs + r);
        hx = ox + dir.x * t;
        hy = oy + dir.y * t;
        hz = oz + dir.z * t;
    }
    const uint32_t* list = nullptr;
    uint32_t count = 0;
    if (hit) list = leaf_lights(s, leaf_nid[sample], count);
    const uint32_t jmax = min(__reduce_max_sync(0xFFFFFFFFu, count), 15u);
    Places pl;
    pl.want(kKindSun, hit);
    const uint32_t direct_bits = want_lights(s, pl, list, count, jmax, hx, hy, hz);
    pl.reserve(g, 0u);
    pl.put(g, 0u, kKindSun, hit, sample, hx, hy, hz, kTMax, -d.sun[0], -d.sun[1], -d.sun[2], 1u);
    put_lights(s, g, pl, 0u, list, jmax, sample, hx, hy, hz);
    if (valid) {
        g.out_words[8u * sample + 4u] = direct_bits;
        g.out_words[8u * sample + 5u] = 0u;
    }
    finish_queue(g);
}

// core/lighting.glsl:16-20 computeAttenuation
__device__ __forceinline__ float attenuation(float dist, float radius) {
    const float att = (radius * radius + 1.0f) / (255.0f * dist * dist);
    return fminf(fmaxf(att - (1.0f / 255.0f), 0.0f), 1.0f);
}

// core/lighting.glsl:22-57 computeLighting (texColor = 1, no shadow ray on the fly)
// and 137-182 computePbrLighting; m = the Material record (12 words).
__device__ void compute_lighting(const float* m, float lcx, float lcy, float lcz, float px, float py, float pz,
                                 float Lx, float Ly, float Lz, float Nx, float Ny, float Nz, float ex, float ey,
                                 float ez, float att, float& ox, float& oy, float& oz) {
    const uint32_t type = __float_as_uint(__ldg(m));
    const float cr = __ldg(m + 4), cg = __ldg(m + 5), cb = __ldg(m + 6);
    if (type == 1u) { ox = cr; oy = cg; oz = cb; return; }            // Material_Emissive
    if (type == 4u) { ox = oy = oz = 0.0f; return; }                  // Material_Transparent
    float rx = 0.f, ry = 0.f, rz = 0.f;
    const float dotL = fminf(fmaxf(dot3(Nx, Ny, Nz, Lx, Ly, Lz), 0.0f), 1.0f);
    if (type == 5u) {                                                 // Material_PBR
        const float metal = __ldg(m + 8);
        float vx = ex - px, vy = ey - py, vz = ez - pz;
        const float vl = sqrtf(dot3(vx, vy, vz, vx, vy, vz));
        vx = vx / vl; vy = vy / vl; vz = vz / vl;
        float hx = vx + Lx, hy = vy + Ly, hz = vz + Lz;
        const float hl = sqrtf(dot3(hx, hy, hz, hx, hy, hz));
        hx = hx / hl; hy = hy / hl; hz = hz / hl;
        const float NoV = fabsf(dot3(Nx, Ny, Nz, vx, vy, vz)) + 1e-5f;
        const float NoL = fminf(fmaxf(dot3(Nx, Ny, Nz, Lx, Ly, Lz), 0.0f), 1.0f);
        const float NoH = fminf(fmaxf(dot3(Nx, Ny, Nz, hx, hy, hz), 0.0f), 1.0f);
        const float LoH = fminf(fmaxf(dot3(Lx, Ly, Lz, hx, hy, hz), 0.0f), 1.0f);
        const float rough = 0.02f * 0.02f;
        const float a2 = rough * rough;
        const float f = (NoH * a2 - NoH) * NoH + 1.0f;
        const float D = a2 / (3.141592f * f * f);
        const float f0x = 0.04f * (1.0f - metal) + cr * metal, f0y = 0.04f * (1.0f - metal) + cg * metal,
                    f0z = 0.04f * (1.0f - metal) + cb * metal;
        const float p5 = powf(1.0f - LoH, 5.0f);
        const float Fx = f0x + (1.0f - f0x) * p5, Fy = f0y + (1.0f - f0y) * p5, Fz = f0z + (1.0f - f0z) * p5;
        const float GGXL = NoV * sqrtf((-NoL * a2 + NoL) * NoL + a2);
        const float GGXV = NoL * sqrtf((-NoV * a2 + NoV) * NoV + a2);
        const float V = 0.5f / (GGXV + GGXL);
        const float DV = D * V;
        const float dx = cr * (1.0f - metal) / 3.141592f, dy = cg * (1.0f - metal) / 3.141592f,
                    dz = cb * (1.0f - metal) / 3.141592f;
        rx = ((dx + Fx * DV) * lcx) * NoL;
        ry = ((dy + Fy * DV) * lcy) * NoL;
        rz = ((dz + Fz * DV) * lcz) * NoL;
    } else if (type == 2u) {                                          // Material_Lambert
        rx = (lcx * dotL) * cr;
        ry = (lcy * dotL) * cg;
        rz = (lcz * dotL) * cb;
    }
    ox = rx * att;
    oy = ry * att;
    oz = rz * att;
}

// baseRaytracingPass.glsl:38-64 fillUvNormal, the normal: barycentric weights of
// the hit point in the hit triangle (record rec) and the interpolated vertex normal.
__device__ __forceinline__ void hit_normal(const SceneView& s, const uint4& rec, float px, float py, float pz,
                                           float& Nx, float& Ny, float& Nz) {
    const uint32_t i0 = rec.x + (rec.y & 0xFFFFu), i1 = rec.x + (rec.y >> 16), i2 = rec.x + (rec.z & 0xFFFFu);
    const float* P = s.pos;
    const float v0x = P[3 * i1] - P[3 * i0], v0y = P[3 * i1 + 1] - P[3 * i0 + 1], v0z = P[3 * i1 + 2] - P[3 * i0 + 2];
    const float v1x = P[3 * i2] - P[3 * i0], v1y = P[3 * i2 + 1] - P[3 * i0 + 1], v1z = P[3 * i2 + 2] - P[3 * i0 + 2];
    const float v2x = px - P[3 * i0], v2y = py - P[3 * i0 + 1], v2z = pz - P[3 * i0 + 2];
    const float d00 = dot3(v0x, v0y, v0z, v0x, v0y, v0z), d01 = dot3(v0x, v0y, v0z, v1x, v1y, v1z);
    const float d11 = dot3(v1x, v1y, v1z, v1x, v1y, v1z);
    const float d20 = dot3(v2x, v2y, v2z, v0x, v0y, v0z), d21 = dot3(v2x, v2y, v2z, v1x, v1y, v1z);
    const float denom = d00 * d11 - d01 * d01;
    const float v = (d11 * d20 - d01 * d21) / denom;
    const float w = (d00 * d21 - d01 * d20) / denom;
    const float u = 1.0f - v - w;
    const float* Nn = s.nrm;
    Nx = (Nn[3 * i0] * u + Nn[3 * i1] * v) + Nn[3 * i2] * w;
    Ny = (Nn[3 * i0 + 1] * u + Nn[3 * i1 + 1] * v) + Nn[3 * i2 + 1] * w;
    Nz = (Nn[3 * i0 + 2] * u + Nn[3 * i1 + 2] * v) + Nn[3 * i2 + 2] * w;
}

// Whether a squared distance is surely beyond a light's radius: the shader's test is
// sqrt(d2) < radius, and the margins are above what the products and the root round by.
__device__ __forceinline__ bool beyond(float d2, float radius) {
    return d2 > (radius * radius) * (1.0f + 1.0f / 1048576.0f) + 1e-37f;
}

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// The first 31 lights (a mask has no bit for more) that reach a warp's hit points, a bit
// each: lane k measures light k from the points' box, by the operations that measure it
// from a point, none of which can come out larger here. Called by whole warps.
__device__ __forceinline__ uint32_t lights_in_reach(const SceneView& s, bool hit, float px, float py, float pz) {
    const float lox = warp_min(hit ? px : INFINITY), loy = warp_min(hit ? py : INFINITY), loz = warp_min(hit ? pz : INFINITY);
    const float hix = -warp_min(hit ? -px : INFINITY), hiy = -warp_min(hit ? -py : INFINITY), hiz = -warp_min(hit ? -pz : INFINITY);
    const uint32_t li = threadIdx.x & 31u;
    bool reach = false;
    if (li < s.num_lights && li < 31u) {
        const float* L = s.lights + 14u * li;
        const float x = __ldg(L + 1), y = __ldg(L + 2), z = __ldg(L + 3);
        const float ax = fmaxf(fmaxf(x - hix, lox - x), 0.0f), ay = fmaxf(fmaxf(y - hiy, loy - y), 0.0f),
                    az = fmaxf(fmaxf(z - hiz, loz - z), 0.0f);
        reach = __float_as_uint(__ldg(L)) == kLightSphere && !beyond(dot3(ax, ay, az, ax, ay, az), __ldg(L + 4));
    }
    return __ballot_sync(0xFFFFFFFFu, reach);
}

// bvhLighting.glsl:42-85 computeLighting, direct part (texColor 1): the lights whose
// shadow-mask bit is clear (evalLighting -> evalSphereLight; an out-of-range light
// adds nothing), then the sun (evalSunLight), summed in the shader's order.
__device__ void direct_lit(const SceneView& s, const float* m, float px, float py, float pz, float Nx, float Ny,
                           float Nz, float ex, float ey, float ez, uint32_t mask, uint32_t reach, const float* sun,
                           const float* sunc, float& lx, float& ly, float& lz) {
    lx = 0.f; ly = 0.f; lz = 0.f;
    for (; reach; reach &= reach - 1u) {
        const uint32_t li = (uint32_t)__ffs((int)reach) - 1u;
        if (mask & (1u << (li + 1u))) continue;
        const float* L = s.lights + 14u * li;
        const float ax = __ldg(L + 1) - px, ay = __ldg(L + 2) - py, az = __ldg(L + 3) - pz, radius = __ldg(L + 4);
        const float d2 = dot3(ax, ay, az, ax, ay, az);
        if (beyond(d2, radius)) continue;
        float dd = sqrtf(d2);
        if (dd < radius) {
            const float Lx = ax / dd, Ly = ay / dd, Lz = az / dd;
            dd = fmaxf(0.01f, dd - __ldg(L + 8));
            float cx, cy, cz;
            compute_lighting(m, __ldg(L + 5), __ldg(L + 6), __ldg(L + 7), px, py, pz, Lx, Ly, Lz, Nx, Ny, Nz, ex, ey,
                             ez, attenuation(dd, radius), cx, cy, cz);
            lx = lx + cx; ly = ly + cy; lz = lz + cz;
        }
    }
    if ((mask & 1u) == 0u) {
        float cx, cy, cz;
        compute_lighting(m, sunc[0], sunc[1], sunc[2], px, py, pz, -sun[0], -sun[1], -sun[2], Nx, Ny, Nz, ex, ey, ez,
                         1.0f, cx, cy, cz);
        lx = lx + cx; ly = ly + cy; lz = lz + cz;
    }
}

// baseRaytracingPass.glsl:81: the colour of a miss, 0.3 * vec3(200, 220, 255) / 255.
__device__ __forceinline__ void sky_colour(float& lx, float& ly, float& lz) {
    lx = (0.3f * 200.0f) / 255.0f;
    ly = (0.3f * 220.0f) / 255.0f;
    lz = (0.3f * 255.0f) / 255.0f;
}

// Lit value of one probe ray: bvhLighting.glsl:42-85 computeLighting with NO_LPF
// (genLightProbField.comp:5), normal from baseRaytracingPass.glsl:38-64, sky
// colour on a miss (baseRaytracingPass.glsl:81).
__global__ void __launch_bounds__(256) k_probe_light(SceneView s, ProbeArgs d, const uint32_t* out_words, float* irr) {
    const uint32_t sample = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = sample < d.np * d.nd;
    uint4 rec = make_uint4(0u, 0u, 0u, __float_as_uint(kTMax));
    float ox = 0.f, oy = 0.f, oz = 0.f, px = 0.f, py = 0.f, pz = 0.f;
    uint32_t mask = 0u;
    if (valid) {
        rec = reinterpret_cast<const uint4*>(out_words)[2u * sample];
        mask = out_words[8u * sample + 4u];
    }
    const float t = __uint_as_float(rec.w);
    const bool hit = t < kTMax;
    if (hit) {
        probe_position(d, d.p0 + sample / d.nd, ox, oy, oz);
        const float4 dir = __ldg(d.dirs + sample % d.nd);
        px = ox + dir.x * t; py = oy + dir.y * t; pz = oz + dir.z * t;
    }
    const uint32_t reach = lights_in_reach(s, hit, px, py, pz);
    if (!valid) return;
    float lx, ly, lz;
    if (!hit) {
        sky_colour(lx, ly, lz);
    } else {
        float Nx, Ny, Nz;
        hit_normal(s, rec, px, py, pz, Nx, Ny, Nz);
        const float* m = s.materials + 12u * (rec.z >> 16);
        direct_lit(s, m, px, py, pz, Nx, Ny, Nz, ox, oy, oz, mask, reach, d.sun, d.sunc, lx, ly, lz);
    }
    irr[3u * sample] = lx;
    irr[3u * sample + 1u] = ly;
    irr[3u * sample + 2u] = lz;
}

// updateLightProbField.comp:33-64: rays summed in order (j-th SH coefficient, r,g,b), x
// 4*pi/N, GLSL mix with the previous FP16 value, stored back as FP16 in storeSH9's channel
// layout; plus the octahedral texels. A block takes kAccumProbes probes, a thread one of
// the 27 sums of one of them, over rays and weights brought to shared memory kAccumRays
// at a time: the sums' orders are fixed, so the chain of additions is what a probe takes,
// and 27 threads a probe fill the GPU where one did not (8,192 probes were 64 blocks:
// 208 us; now 46).
constexpr uint32_t kAccumProbes = 8, kAccumRays = 64, kAccumThreads = 224;
__global__ void __launch_bounds__(kAccumThreads) k_probe_accum(ProbeArgs d, const float* irr, uint16_t* sh16, float* sh32,
                                                               float* octa, uint32_t side) {
    __shared__ float lit[kAccumProbes][3 * kAccumRays];
    __shared__ float weight[9 * kAccumRays];
    const uint32_t first = blockIdx.x * kAccumProbes, probes = min(kAccumProbes, d.np - first), nd = d.nd;
    const uint32_t mine = threadIdx.x / 27u, q = threadIdx.x % 27u, j = q / 3u, c = q % 3u;
    const float* L = irr + 3ull * first * nd;
    float acc = 0.0f;
    for (uint32_t r0 = 0; r0 < nd; r0 += kAccumRays) {
        const uint32_t n = min(kAccumRays, nd - r0);
        for (uint32_t i = threadIdx.x; i < probes * 3u * n; i += kAccumThreads) {
            const uint32_t p = i / (3u * n), k = i - p * 3u * n;
            lit[p][k] = L[3ull * (p * (uint64_t)nd + r0) + k];
        }
        for (uint32_t i = threadIdx.x; i < 9u * n; i += kAccumThreads) weight[i] = __ldg(d.basis + 9u * r0 + i);
        __syncthreads();
        if (mine < probes)
            for (uint32_t r = 0; r < n; ++r) acc = acc + lit[mine][3u * r + c] * weight[9u * r + j];
        __syncthreads();
    }
    if (mine < probes) {
        const float norm = (4.0f * 3.14159265358979323846f) / (float)nd;
        uint32_t cx, cy, cz;
        probe_coord(d.p0 + first + mine, d.res, cx, cy, cz);
        const uint64_t texel = ((uint64_t)cz * d.res[1] + cy) * d.res[0] + cx;
        const uint64_t img = (uint64_t)d.res[0] * d.res[1] * d.res[2];
        const float a = d.hyst;
        const uint32_t image = j == 0u ? 0u : (j <= 4u ? 1u + 2u * c : 2u + 2u * c);
        const uint32_t ch = j == 0u ? c : (j <= 4u ? j - 1u : j - 5u);
        uint16_t* h = sh16 + 4ull * (image * img + texel) + ch;
        const float prev = __half2float(__ushort_as_half(*h));
        const float nw = prev * (1.0f - a) + (acc * norm) * a;
        *h = __half_as_ushort(__float2half_rn(nw));
        if (sh32) sh32[27ull * (first + mine) + q] = nw;
        if (q == 0u) sh16[4ull * texel + 3] = 0;   // image 0 alpha (storeSH9 writes 0)
    }
    if (octa) {
        const uint32_t step = side / 8u;
        const float inv = 1.0f / (float)(step * step);
        for (uint32_t i = threadIdx.x; i < probes * 192u; i += kAccumThreads) {
            const uint32_t p = i / 192u, o = i % 192u, t = o / 3u, ch = o % 3u, tx = t % 8u, ty = t / 8u;
            const float* Lp = L + 3ull * p * nd;
            float sum = 0.f;
            for (uint32_t jj = ty * step; jj < (ty + 1u) * step; ++jj)
                for (uint32_t ii = tx * step; ii < (tx + 1u) * step; ++ii) sum = sum + Lp[3u * (jj * side + ii) + ch];
            octa[192ull * (first + p) + o] = sum * inv;
        }
    }
}

// ------------------------------------------------------------ camera lighting step
// fetchSH_inline.glsl:82-118 sampleSH9 with the probe mask (bit x + 2y + 4z set = that
// corner masked): GLSL mix, a * (1 - f) + b * f, of each pair along x, then y, then z; of
// a pair with one side masked the other side as it is; of a pair with both, the second.
// Here every pair is one product sum whatever the mask: a masked side's value is -0 and
// its weight 0, the other's weight 1, and x * 1 + -0 * 0 is x for every x (-0 * 0 is -0,
// the sum's neutral element); all corners masked is the shader's last corner alone. So
// the mask costs seven pairs of weights a pixel instead of seven selects a channel, and
// the cells' lower and upper half (corners q and q + 4) go through packed operations,
// whose halves round as the scalar ones do. The sum is a packed FMA by a `one` that the
// compiler can't see: it contracts a packed product and a packed add, whatever the flags.
// (Two channels to a packed operation needs each weight twice in registers: 97 us for the
// 1080p step of k_shade_camera's comment, against 90 us.)
struct Lerp { float a, b; };
__device__ __forceinline__ Lerp lerp_weights(bool has_a, bool has_b, float f) {
    return {has_a && has_b ? 1.0f - f : (has_b && !has_a ? 0.0f : 1.0f), has_a && has_b ? f : (has_b && !has_a ? 1.0f : 0.0f)};
}
struct Lerp2 { uint64_t a, b; };
__device__ __forceinline__ Lerp2 both(const Lerp& lo, const Lerp& hi) { return {pack2f(lo.a, hi.a), pack2f(lo.b, hi.b)}; }
__device__ __forceinline__ uint64_t lerp2(uint64_t a, uint64_t b, const Lerp2& w, uint64_t one) {
    return fma2(mul2(a, w.a), one, mul2(b, w.b));
}
__device__ __forceinline__ float half_of(uint32_t h, int hi) {
    return __half2float(__ushort_as_half((unsigned short)(hi ? h >> 16 : h & 0xFFFFu)));
}

// bvhLighting.glsl:24-40 computeLPFLighting with USE_LPF_MASK: probe-grid uvw
// (lightprobHelpers.glsl:10-14,71-77), masked SH9 sample of the 7 RGBA16F images
// (fetchSH_inline.glsl:6-31 channel layout), evalSH (lightprobHelpers.glsl:90-101)
// and computeIndirectLighting (core/lighting.glsl:59-74, texColor 1).
__device__ void lpf_lit(const tim_rt_pass_data& pd, const uint2* sh16, const float* m, float px, float py, float pz,
                        float Nx, float Ny, float Nz, uint32_t mask, float one, float& lx, float& ly, float& lz) {
    const uint32_t rx = pd.lpfResolution[0], ry = pd.lpfResolution[1], rz = pd.lpfResolution[2];
    const float sx = (pd.sceneMaxExtent[0] - pd.sceneMinExtent[0]) / (float)rx;
    const float sy = (pd.sceneMaxExtent[1] - pd.sceneMinExtent[1]) / (float)ry;
    const float sz = (pd.sceneMaxExtent[2] - pd.sceneMinExtent[2]) / (float)rz;
    float u = (px - pd.sceneMinExtent[0]) / sx - 0.5f;
    float v = (py - pd.sceneMinExtent[1]) / sy - 0.5f;
    float w = (pz - pd.sceneMinExtent[2]) / sz - 0.5f;
    u = fminf(fmaxf(u, 0.0f), (float)rx - 1.0f);
    v = fminf(fmaxf(v, 0.0f), (float)ry - 1.0f);
    w = fminf(fmaxf(w, 0.0f), (float)rz - 1.0f);
    // min(int(uvw), res - 2) in GLSL's int -> uint conversion
    const uint32_t ix = min((uint32_t)(int)u, rx - 2u), iy = min((uint32_t)(int)v, ry - 2u),
                   iz = min((uint32_t)(int)w, rz - 2u);
    const float fx = u - (float)(int)ix, fy = v - (float)(int)iy, fz = w - (float)(int)iz;
    if ((mask & 0xFFu) == 0xFFu) mask = 0x7Fu;
    bool on[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) on[q] = !(mask & (1u << q));
    const Lerp2 wx0 = both(lerp_weights(on[0], on[1], fx), lerp_weights(on[4], on[5], fx));
    const Lerp2 wx1 = both(lerp_weights(on[2], on[3], fx), lerp_weights(on[6], on[7], fx));
    const Lerp2 wy = both(lerp_weights(on[0] || on[1], on[2] || on[3], fy), lerp_weights(on[4] || on[5], on[6] || on[7], fy));
    const Lerp wz = lerp_weights(on[0] || on[1] || on[2] || on[3], on[4] || on[5] || on[6] || on[7], fz);
    const uint64_t img = (uint64_t)rx * ry * rz, one2 = pack2f(one, one);
    const uint2* corner = sh16 + ((uint64_t)iz * ry + iy) * rx + ix;
    auto sample = [&](uint32_t k, float (&ch)[4]) {
        uint2 h[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            h[q] = make_uint2(0x80008000u, 0x80008000u);   // -0
            if (on[q]) h[q] = __ldg(corner + k * img + ((uint64_t)((q >> 2) & 1) * ry + ((q >> 1) & 1)) * rx + (q & 1));
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
            uint64_t v[4];   // corner q and the one above it
#pragma unroll
            for (int q = 0; q < 4; ++q)
                v[q] = pack2f(half_of(cc < 2 ? h[q].x : h[q].y, cc & 1), half_of(cc < 2 ? h[q + 4].x : h[q + 4].y, cc & 1));
            float z0, z1;
            unpack2f(lerp2(lerp2(v[0], v[1], wx0, one2), lerp2(v[2], v[3], wx1, one2), wy, one2), z0, z1);
            ch[cc] = z0 * wz.a + z1 * wz.b;
        }
    };
    const float c1 = 0.429043f, c2 = 0.511664f, c3 = 0.743125f, c4 = 0.886227f, c5 = 0.247708f;
    float band0[4], L[3];
    sample(0u, band0);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        // SH9Color.w[j] from the storeSH9 layout: w0 = image 0; w1..4 = images 1/3/5, w5..8 = images 2/4/6
        float a[4], b[4];
        sample(1u + 2u * c, a);
        sample(2u + 2u * c, b);
        const float w0 = c == 0 ? band0[0] : (c == 1 ? band0[1] : band0[2]);
        const float w1 = a[0], w2 = a[1], w3 = a[2], w4 = a[3], w5 = b[0], w6 = b[1], w7 = b[2], w8 = b[3];
        // SH_Y00 0, Y11 1, Y10 2, Y1_1 3, Y21 4, Y2_1 5, Y2_2 6, Y20 7, Y22 8 (lightprob/lightprob.glsl)
        const float t1 = (c1 * (Nx * Nx - Ny * Ny)) * w8;
        const float t2 = ((c3 * w7) * Nz) * Nz;
        const float t3 = c4 * w0;
        const float t4 = c5 * w7;
        const float t5 = (2.0f * c1) * (((w6 * Nx) * Ny + (w4 * Nx) * Nz) + (w5 * Ny) * Nz);
        const float t6 = (2.0f * c2) * ((w1 * Nx + w3 * Ny) + w2 * Nz);
        const float l = ((((t1 + t2) + t3) - t4) + t5) + t6;
        if (c == 0) L[0] = l; else if (c == 1) L[1] = l; else L[2] = l;
    }
    const uint32_t type = __float_as_uint(__ldg(m));
    const float cr = __ldg(m + 4), cg = __ldg(m + 5), cb = __ldg(m + 6);
    const float pi = 3.14159265359f;   // TIM_PI, core/math.glsl:4
    if (type == 5u) {                  // Material_PBR
        const float k = 1.0f - __ldg(m + 8);
        lx = ((k * cr) * L[0]) / pi; ly = ((k * cg) * L[1]) / pi; lz = ((k * cb) * L[2]) / pi;
    } else if (type == 2u) {           // Material_Lambert
        lx = (L[0] * cr) / pi; ly = (L[1] * cg) / pi; lz = (L[2] * cb) / pi;
    } else {
        lx = ly = lz = 0.0f;
    }
}

// cameraPass.comp:78-88, the lighting step (RayTracingPass::lightingPass,
// raytracingPass.cpp:113-135: USE_LPF, USE_LPF_MASK). One thread per output pixel, a warp
// an 8 x 4 tile (few lights reach it, and its records, texels and image rows are whole
// sectors); the pixel's ray is the tracing step's (cameraPass.comp:46-56), output row 0
// is never reached by the reference's dispatch and is written as 0.
// Bound by instruction issue (78% of the cycles; 1,200 instructions a warp, half of them
// the probe field's 27 interpolated channels): 1920 x 1080, 16 lights, 12^3 probes took
// 149 us (72 without the probe field) with a row of 32 pixels a warp, every light measured
// by every pixel and the mask's selects in each channel; 90 us (41) now. Four blocks an SM
// (64 registers, a few spilled) against three: 96 us (49); five: 105 us (38).
__global__ void __launch_bounds__(256, 4) k_shade_camera(SceneView s, tim_rt_pass_data pd, uint32_t flags,
                                                         const uint4* tracing, const uint2* sh16, uint2* out16,
                                                         float* out32, float one) {
    const uint32_t W = pd.frameSize[0], H = pd.frameSize[1];
    const uint32_t across = (W + 31u) / 32u, warp = threadIdx.x / 32u, lane = threadIdx.x & 31u;
    const uint32_t px = blockIdx.x % across * 32u + (warp & 3u) * 8u + (lane & 7u);
    const uint32_t py = blockIdx.x / across * 8u + (warp >> 2) * 4u + (lane >> 3);
    const uint64_t pix = (uint64_t)py * W + px;
    const bool valid = px < W && py < H, reached = valid && py != 0u;
    const float ex = pd.cameraPos[0], ey = pd.cameraPos[1], ez = pd.cameraPos[2];
    uint4 rec = make_uint4(0u, 0u, 0u, __float_as_uint(kTMax)), masks = rec;
    float hx = 0.f, hy = 0.f, hz = 0.f;
    if (reached) {
        rec = __ldg(tracing + 2u * pix);
        masks = __ldg(tracing + 2u * pix + 1u);
    }
    const float t = __uint_as_float(rec.w);
    const bool hit = t < kTMax;
    if (hit) {
        const uint32_t ngy16 = 16u * ((H + 15u) / 16u);
        float dx, dy, dz;
        camera_ray(pd, px, ngy16 - py, dx, dy, dz);
        hx = ex + dx * t; hy = ey + dy * t; hz = ez + dz * t;
    }
    const uint32_t reach = lights_in_reach(s, hit, hx, hy, hz);
    if (!valid) return;
    float lx = 0.f, ly = 0.f, lz = 0.f;
    if (hit) {
        float Nx, Ny, Nz;
        hit_normal(s, rec, hx, hy, hz, Nx, Ny, Nz);
        const float* m = s.materials + 12u * (rec.z >> 16);
        direct_lit(s, m, hx, hy, hz, Nx, Ny, Nz, ex, ey, ez, masks.x, reach, pd.sunDir, pd.sunColor, lx, ly, lz);
        if (!(flags & TIM_RT_SHADE_NO_LPF)) {
            float ix, iy, iz;
            lpf_lit(pd, sh16, m, hx, hy, hz, Nx, Ny, Nz, masks.y, one, ix, iy, iz);
            lx = lx + ix; ly = ly + iy; lz = lz + iz;
        }
    } else if (reached) {
        sky_colour(lx, ly, lz);
    }
    const uint32_t hr = __half_as_ushort(__float2half_rn(lx)), hg = __half_as_ushort(__float2half_rn(ly));
    const uint32_t hb = __half_as_ushort(__float2half_rn(lz));
    const uint32_t ha = reached ? 0x3C00u : 0u;   // alpha 1
    out16[pix] = make_uint2(hr | (hg << 16), hb | (ha << 16));
    if (out32) {
        out32[3u * pix] = lx;
        out32[3u * pix + 1u] = ly;
        out32[3u * pix + 2u] = lz;
    }
}

cudaError_t launch_shade(const SceneView& s, const tim_rt_pass_data& pd, uint32_t flags, const uint32_t* tracing,
                         const uint16_t* sh16, uint16_t* out16, float* out32, cudaStream_t stream) {
    const uint64_t blocks = ((uint64_t)pd.frameSize[0] + 31u) / 32u * (((uint64_t)pd.frameSize[1] + 7u) / 8u);
    if (blocks == 0) return cudaSuccess;
    k_shade_camera<<<(unsigned)blocks, 256, 0, stream>>>(
        s, pd, flags, reinterpret_cast<const uint4*>(tracing), reinterpret_cast<const uint2*>(sh16),
        reinterpret_cast<uint2*>(out16), out32, 1.0f);
    return cudaGetLastError();
}

cudaError_t launch_probes(const SceneView& s, const ProbeArgs& d, uint32_t* out, uint32_t* leaf_nid, tim_rt_ray* q_rays,
                          uint32_t* q_pixel, uint32_t* counters, uint32_t* err, float* irr, uint16_t* sh16, float* sh32,
                          float* octa, uint32_t side, cudaStream_t stream, const LaunchConfig& cfg) {
    const uint32_t n = d.np * d.nd;
    ProbePolicy PP{d, reinterpret_cast<uint4*>(out), leaf_nid};
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[0], stream);
    LaunchConfig pcfg = cfg;
    pcfg.wide = cfg.wide && !cfg.primary_binary;
    PP.d.trace_dir_major = d.trace_dir_major && (pcfg.wide || !use_walk(s, pcfg));
    cudaError_t e = use_walk(s, pcfg) ? launch_rays<false>(s, PP, n, counters + 0, err, stream, pcfg)
                                      : launch_general(s, PP, n, counters + 0, err, stream, pcfg);
    if (e != cudaSuccess) return e;
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[1], stream);
    GenParams g{};
    g.out_words = out;
    g.q_rays = q_rays;
    g.q_pixel = q_pixel;
    QueueBands qb{};
    qb.n = 1;
    qb.cap[0] = n;
    queue_counters(counters, qb, nullptr, use_walk(s, cfg), g);
    k_probe_gen<<<(n + 255u) / 256u, 256, 0, stream>>>(s, d, g, leaf_nid);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[2], stream);
    LaunchConfig cfg2 = cfg;
    if (cfg.stats) cfg2.stats = cfg.stats + 8;
    e = launch_secondary(s, g, counters, err, stream, cfg2, false);
    if (cfg.phase_ev) cudaEventRecord(cfg.phase_ev[3], stream);
    if (e != cudaSuccess) return e;
    k_probe_light<<<(n + 255u) / 256u, 256, 0, stream>>>(s, d, out, irr);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_probe_accum<<<(d.np + kAccumProbes - 1u) / kAccumProbes, kAccumThreads, 0, stream>>>(d, irr, sh16, sh32, octa, side);
    return cudaGetLastError();
}

}  // namespace timrt
