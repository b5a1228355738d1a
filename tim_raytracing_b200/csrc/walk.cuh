// walk.cuh -- the persistent kernel for rays of one kind (k_walk) and its launcher, for the
// single-scene launches (trace.cu) and the batched ones (multi.cu).
#pragma once
#include "common.cuh"
#include "kernels.h"
#include "trace_any.cuh"
#include "trace_pair.cuh"
#include "trace_quant.cuh"

namespace timrt {

// Whether a policy wants its finished() hook called by the whole warp after each
// round of stores.
template <class P, class = void>
struct finishes { static constexpr bool value = false; };
template <class P>
struct finishes<P, decltype((void)P::kFinishes)> { static constexpr bool value = P::kFinishes; };

// Whether a policy traces only the items that keeps() tells of its batch.
template <class P, class = void>
struct filters { static constexpr bool value = false; };
template <class P>
struct filters<P, decltype((void)P::kFilters)> { static constexpr bool value = P::kFilters; };

// Whether each ray of a policy names its own scene (views[st.view]).
template <class P, class = void>
struct many_scenes { static constexpr bool value = false; };
template <class P>
struct many_scenes<P, decltype((void)P::kManyScenes)> { static constexpr bool value = P::kManyScenes; };

// The work items of a launch: the policy's own count, or the launch's.
template <class P, class = void>
struct counts_items { static constexpr bool value = false; };
template <class P>
struct counts_items<P, decltype((void)&P::items)> { static constexpr bool value = true; };
template <class Policy>
__device__ __forceinline__ uint32_t items_of(const Policy& P, uint32_t n) {
    if constexpr (counts_items<Policy>::value) return P.items();
    else return n;
}

// Hands the items of a batch that a filtering policy (filters<Policy>) keeps to the
// idle lanes of a warp: `batch` items (up to 32) at a time are looked at, those kept wait in `pool`
// (32 words of shared memory a warp) until lanes take them. start(item) is called by
// the lanes that got one; sets exhausted once the batch is used up.
template <class Policy, class Start>
__device__ __forceinline__ void refill_filtered(const Policy& P, uint32_t n, uint32_t* counter, uint32_t* pool,
                                                uint32_t need, uint32_t batch, uint32_t& used, uint32_t& have,
                                                bool& exhausted, Start start) {
    const uint32_t lane = threadIdx.x & 31u;
    while (need) {
        if (used == have) {
            uint32_t base = 0;
            if (lane == 0u) base = atomicAdd(counter, batch);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (base >= n) {
                exhausted = true;
                return;
            }
            const uint32_t item = base + lane;
            const bool mine = lane < batch && item < n && P.keeps(item);
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, mine);
            if (mine) pool[__popc(m & lanemask_lt())] = item;
            __syncwarp();
            used = 0;
            have = (uint32_t)__popc(m);
            continue;
        }
        const uint32_t r = (uint32_t)__popc(need & lanemask_lt());
        const bool take = ((need >> lane) & 1u) && r < have - used;
        if (take) start(pool[used + r]);
        __syncwarp();
        used = min(have, used + (uint32_t)__popc(need));
        need &= ~__ballot_sync(0xFFFFFFFFu, take);
    }
}

// Shared-memory words a thread of k_walk has beside its stack: the ray's origin and
// direction, in batched launches what names its job and scene, in the 8-wide form its
// tmax, and two of its warp's.
template <class Policy, bool QUANT>
constexpr int walk_words = (many_scenes<Policy>::value ? 11 : 8) + (QUANT ? 1 : 0);
// A warp's leaves are spread over its lanes up to this many triangles (two rounds; a leaf
// of four on each lane's own takes four). 1M mixed rays / the 16-scene batch / probe rays:
// 0.463 / 2.11 / 1.00 ms with 32, 0.453 / 2.01 / 0.97 with 64, 0.453 / 1.98 / 0.96 with
// 96, which costs the bounce and camera rays 2 %.
constexpr uint32_t kSpreadMost = 64u;
// A ray alone on its warp waits for no other's loads and leaves: launches of few rays are
// bound by that latency, not by the GPU's width. Closest-hit rays in the 100K-triangle
// scene, 32 rays a warp / spread: 100 rays 64 / 44 us, 1,000 87 / 64, 4,000 106 / 92,
// 16,000 140 / 134; any-hit 53 / 42, 66 / 49, 77 / 70, 100 / 98; 64,000 (14 lanes) no less.
constexpr uint32_t kFewLanes = 8u;
// Threads per SM the registers are cut to. The batches' kernels hold more per ray and
// their rays miss the L1 most: 3 blocks without spills instead of 4 with (1M mixed rays
// 0.427 against 0.451 ms, the 16-scene batch 2.26 against 2.36); the others 4 blocks
// (camera rays 0.33 against 0.36 ms, probe rays 1.02 against 1.09). In the 8-wide form
// the closest-hit rays take 3 (secondary rays of a frame 1.42 -> 1.39 ms).
template <class Policy, bool ANY, bool QUANT>
constexpr int walk_threads = filters<Policy>::value || (QUANT && !ANY) ? 768 : 1024;

// Rays of one kind on their own tree: in the binary form any-hit rays on the 4-wide one
// (trace_any.cuh), closest-hit rays on the binary one's child pairs (trace_pair.cuh); in
// the 8-wide form (QUANT) both on the quantised one (trace_quant.cuh). The same
// persistent loop, with the ray's place in st.node alone -- an inner node, a leaf, or
// kAnyIdle, which is also the lowest word of its stack, so that popping it ends the
// walk. sdepth: stack words per thread, as many as any ray needs.
//
// A batch of both kinds is two launches (kPairFirst, kPairSecond) that may overlap: the
// first lets the second start as soon as its own blocks leave room, so that the second's
// rays fill the first's tail; neither reads what the other writes, and the second ends
// only after the first has.
constexpr int kAlone = 0, kPairFirst = 1, kPairSecond = 2;
template <int BLOCK, bool ANY, bool QUANT, class Policy>
__global__ void __launch_bounds__(BLOCK, walk_threads<Policy, ANY, QUANT> / BLOCK) k_walk(SceneView s, Policy P, uint32_t n_static, uint32_t* counter,
                                                              uint32_t* err, int sdepth, int knobs) {
    extern __shared__ uint32_t stack_mem[];
    // knobs: refill threshold (bits 0..7), phase-switch threshold (bits 8..15), role in a pair (bits 16..)
    if ((knobs >> 16) == kPairFirst) cudaTriggerProgrammaticLaunchCompletion();
    const uint32_t phase_sw = (uint32_t)(knobs >> 8) & 0xFFu;
    uint32_t* stk = stack_mem + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t n = items_of(P, n_static);
    // Few rays are spread over all warps, up to kFewLanes lanes of each taking part (the
    // rest help with leaf triangles); one launch of a pair takes half of the blocks, which
    // leaves room for the other's rays.
    const uint32_t blocks = (knobs >> 16) == kAlone ? gridDim.x : (gridDim.x + 1u) / 2u, warps = blocks * (BLOCK / 32);
    const bool few = n <= kFewLanes * warps;
    const uint32_t lanes = few ? max(1u, (n + warps - 1u) / warps) : 32u;
    const uint32_t all = lanes == 32u ? 0xFFFFFFFFu : (1u << lanes) - 1u;
    const int refill_min = min(knobs & 0xFF, (int)lanes);
    uint32_t* org = stk + (size_t)sdepth * BLOCK;   // the ray's origin and direction
    uint32_t* dir = org + 3 * BLOCK;
    uint32_t* own = dir + 3 * BLOCK;                 // many_scenes<Policy>: the ray's job, its place there, its scene
    uint32_t* tab = stack_mem + (size_t)(sdepth + walk_words<Policy, QUANT> - 2) * BLOCK + (threadIdx.x & ~31u);   // of the warp
    uint32_t* res = tab + BLOCK;
    uint32_t* far = own + (many_scenes<Policy>::value ? 3 * BLOCK : 0);   // QUANT: the ray's tmax
    uint32_t* pool = stack_mem + (size_t)(sdepth + walk_words<Policy, QUANT>) * BLOCK + (threadIdx.x & ~31u);   // filters<Policy> only
    uint32_t used = 0, have = 0;
    // Where few lanes hold leaves at a time -- closest-hit rays (9 to 14 of 32), batches in
    // any order (5) -- their triangles are spread over the warp. The any-hit rays of frames
    // and probe fields (16 to 22 lanes) are faster on their own lanes, 0.92 against 0.97 ms.
    constexpr bool kSpread = !ANY || filters<Policy>::value;
    const uint32_t bottom = (uint32_t)__cvta_generic_to_shared(stk);
    const uint32_t near = four_near(bottom, sdepth, (int)s.depth4, 4u * BLOCK);   // any-hit rays (four_stack.h)

    TravState st;
    st.node = kAnyIdle;
    bool pending = false, exhausted = few && blockIdx.x >= blocks;
    uint32_t idx = 0;
    stk[0] = kAnyIdle;
    auto scene = [&]() -> const SceneView& {
        if constexpr (many_scenes<Policy>::value) return P.views[own[2 * BLOCK]];
        else return s;
    };
    auto start = [&](uint32_t item) {
        idx = item;
        if (P.load(s, idx, st)) {
            if constexpr (many_scenes<Policy>::value) {
                own[0] = st.slot;
                own[BLOCK] = st.slot2;
                own[2 * BLOCK] = st.view;
            }
            if constexpr (QUANT) {
                *far = __float_as_uint(st.t);
                quant_init<ANY>(st, bottom);
                st.refs = reinterpret_cast<const char*>(scene().wnodes);
            } else if (ANY) any_init(scene(), st, bottom);
            else pair_init(scene(), st, bottom);
            put3<BLOCK>(org, st.r.ox, st.r.oy, st.r.oz);
            put3<BLOCK>(dir, st.r.dx, st.r.dy, st.r.dz);
            pending = true;
        } else {
            P.skip(idx);
        }
    };
    for (;;) {
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, st.node == kAnyIdle) & all;
        if (idle && (exhausted || __popc(idle) >= refill_min || idle == all)) {
            const bool stored = pending && st.node == kAnyIdle;
            if (stored) {
                pending = false;
                st.any = ANY;
                if constexpr (many_scenes<Policy>::value) {
                    st.slot = own[0];
                    st.slot2 = own[BLOCK];
                }
                if (ANY) get3<BLOCK>(org, st.r.ox, st.r.oy, st.r.oz);
                get3<BLOCK>(dir, st.r.dx, st.r.dy, st.r.dz);
                if constexpr (QUANT) {
                    st.t0 = __uint_as_float(*far);
                    quant_finish<ANY>(scene(), st, P.wants_bary(st), err);
                } else if (ANY) any_finish_or_walk(scene(), st, err);
                else pair_finish(scene(), st, P.wants_nid(st), P.wants_bary(st));
                P.store(s, idx, st, st.t);   // an any-hit ray's t stays its tmax
            }
            if constexpr (finishes<Policy>::value) P.finished(stored, st.slot2);
            if (exhausted) {
                if (idle == all) break;
            } else if constexpr (filters<Policy>::value) {
                refill_filtered(P, n, counter, pool, idle, lanes, used, have, exhausted, start);
            } else {
                const int leader = __ffs(idle) - 1;
                uint32_t base = 0;
                if ((int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(idle));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if ((uint64_t)base + (uint32_t)__popc(idle) >= n) exhausted = true;
                const uint32_t my = base + __popc(idle & lanemask_lt());
                if (((idle >> lane) & 1u) && my < n) start(my);
            }
        }
        for (;;) {   // node rounds (see plain_step_warp)
            const uint32_t nm = __ballot_sync(0xFFFFFFFFu, (int)st.node >= 0);
            if (nm == 0u) break;
            // the threshold is of 32 lanes under way: of fewer, the same part (against a fixed
            // count: 1M mixed rays 0.44 / 0.49 ms, the 16-scene batch 2.15 / 2.32)
            const uint32_t visiting = (uint32_t)__popc(nm);
            if (visiting <= phase_sw) {
                const uint32_t leaves = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, (int)st.node < 0 && st.node != kAnyIdle));
                if (leaves && 32u * visiting <= phase_sw * (visiting + leaves)) break;
            }
            if ((int)st.node >= 0) {
                const char* refs = many_scenes<Policy>::value ? st.refs
                                   : QUANT                    ? reinterpret_cast<const char*>(s.wnodes)
                                   : ANY                      ? four_refs(s)
                                                              : pair_refs(s);
                if (QUANT) quant_advance<BLOCK, ANY>(st, refs, bottom);
                else if (ANY) any_advance<BLOCK>(st, refs, near, bottom, sdepth);
                else pair_advance<BLOCK>(st, refs, dir);
            }
        }
        // leaves: their triangles one by one on their own lanes, or, where few lanes hold
        // one, spread over all lanes
        const bool leaf = (int)st.node < 0 && st.node != kAnyIdle;
        uint32_t first = 0, cnt = 0;
        if (leaf) cnt = QUANT ? quant_leaf(scene(), st.node, first) : leaf_ref(scene(), st.node, first);
        uint32_t incl = cnt, total = 0xFFFFFFFFu;
        if constexpr (kSpread) {
#pragma unroll
            for (uint32_t k = 1; k < 32u; k <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, k);
                if (lane >= k) incl += v;
            }
            total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        }
        bool over = false;   // an any-hit ray has its hit
        if (total > kSpreadMost) {
            if (leaf) {
                Ray r{st.r.ox, st.r.oy, st.r.oz, 0.f, 0.f, 0.f};
                if (ANY) get3<BLOCK>(org, r.ox, r.oy, r.oz);
                get3<BLOCK>(dir, r.dx, r.dy, r.dz);
                over = QUANT ? quant_triangles<ANY>(scene().wtris, st, r, first, cnt, !P.wants_nid(st))
                             : leaf_triangles<ANY>(scene().ptris, st, r, first, cnt);
            }
        } else if (kSpread && total) {
            const uint32_t excl = incl - cnt, owners = __ballot_sync(0xFFFFFFFFu, cnt != 0u);
            if (cnt) tab[__popc(owners & lanemask_lt())] = lane;
            __syncwarp();
            for (uint32_t b = 0; b < total; b += 32u) {
                // place b + lane of the triangles in lane order belongs to the last owner that starts at or before it
                const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, cnt && excl >= b && excl - b < 32u ? 1u << (excl - b) : 0u);
                const uint32_t before = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, cnt && excl < b));
                const bool mine = b + lane < total;
                const uint32_t owner = tab[mine ? before + (uint32_t)__popc(starts & (lanemask_lt() | 1u << lane)) - 1u : 0u];
                const uint32_t tri = __shfl_sync(0xFFFFFFFFu, first - excl, owner) + b + lane;
                const float tmax = __shfl_sync(0xFFFFFFFFu, st.t, owner);
                float t = -1.0f;
                if (mine) {
                    const uint32_t shift = owner - lane;   // the owner's column of the shared words
                    Ray r;
                    get3<BLOCK>(org + (int)shift, r.ox, r.oy, r.oz);
                    get3<BLOCK>(dir + (int)shift, r.dx, r.dy, r.dz);
                    const float4* tp = QUANT ? s.wtris : s.ptris;
                    if constexpr (many_scenes<Policy>::value) {
                        const SceneView& view = P.views[own[2 * BLOCK + (int)shift]];
                        tp = QUANT ? view.wtris : view.ptris;
                    }
                    tp += 3ull * tri;
                    const float4 A = __ldg(tp), B = __ldg(tp + 1), C = __ldg(tp + 2);
                    float u, v;
                    t = collide_triangle_e(r, A.x, A.y, A.z, B.x, B.y, B.z, C.x, C.y, C.z, tmax, u, v);
                }
                const uint32_t hits = __ballot_sync(0xFFFFFFFFu, t > 0.0f);
                if (hits) {
                    if (!ANY) {
                        res[lane] = __float_as_uint(t);
                        __syncwarp();
                    }
                    // the owner's places in this round, in the leaf's order
                    const uint32_t lo = excl > b ? excl - b : 0u, hi = incl > b ? incl - b : 0u;
                    uint32_t m = cnt && lo < 32u ? hits & (0xFFFFFFFFu << lo) & (hi >= 32u ? 0xFFFFFFFFu : (1u << hi) - 1u) : 0u;
                    if (ANY) {
                        if (m && !over) {
                            over = true;
                            st.nid = first - excl + b + (uint32_t)__ffs(m) - 1u;
                        }
                    } else {
                        for (; m; m &= m - 1u) {
                            const uint32_t k = (uint32_t)__ffs(m) - 1u;
                            const float tk = __uint_as_float(res[k]);
                            if constexpr (QUANT) {
                                if (tk < st.t) quant_hit(scene().wtris, st, first - excl + b + k, tk, !P.wants_nid(st));
                            } else if (tk < st.t) {   // the rule triangle by triangle, as leaf_triangles has it
                                st.t = tk - kOffsetRayCollision;
                                st.nid = first - excl + b + k;
                                st.hit = true;
                            }
                        }
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
        }
        if (leaf) {
            if (ANY && over) {
                st.hit = true;
                st.node = kAnyIdle;
            } else if constexpr (QUANT) {
                const uint32_t rest = st.node & (st.node - 1u);
                if (rest & 0xFFu) st.node = rest;
                else quant_next<BLOCK, ANY>(st, bottom);
            } else {
                st.node = stack_pop<BLOCK>(st.top);
            }
        }
    }
    if ((knobs >> 16) == kPairSecond) cudaGridDependencySynchronize();
}

// One word per stack entry, and a filtering policy's 32 words a warp of items not yet handed out.
template <int BLOCK, class Policy>
constexpr size_t stack_bytes(int depth) {
    return sizeof(uint32_t) * (size_t)(depth + (filters<Policy>::value ? 1 : 0)) * BLOCK;
}

// Grid of a persistent kernel: as many resident blocks as the occupancy
// calculator allows on every SM for this stack depth (cached per device and depth).
template <int BLOCK, class Policy, class K>
static int grid_of(GridCache& cache, K* kernel, int depth, int max_depth) {
    return cache.get(depth, [=](int dev) {
        int sms = 0, per = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stack_bytes<BLOCK, Policy>(max_depth));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, BLOCK, stack_bytes<BLOCK, Policy>(depth));
        return (sms > 0 ? sms : 1) * (per > 0 ? per : 1);
    });
}

static_assert(kAnyStack <= kWalkStack, "one limit for all walks");

template <int BLOCK, bool ANY, bool QUANT, class Policy>
static cudaError_t launch_walk_block(const SceneView& s, const Policy& P, uint32_t n_static, uint32_t* counter,
                                     uint32_t* err, int depth, int knobs, int role, int share, cudaStream_t stream) {
    static GridCache cache;
    static_assert(walk_words<Policy, QUANT> <= kWalkBeside, "GridCache counts on it");
    const int words = depth + walk_words<Policy, QUANT>;
    const int grid = grid_of<BLOCK, Policy>(cache, k_walk<BLOCK, ANY, QUANT, Policy>, words, kWalkStack + walk_words<Policy, QUANT>);
    cudaLaunchConfig_t lc{};
    lc.gridDim = dim3(share > 1 && grid >= share ? grid / share : grid);
    lc.blockDim = dim3(BLOCK);
    lc.dynamicSmemBytes = stack_bytes<BLOCK, Policy>(words);
    lc.stream = stream;
    cudaLaunchAttribute at{};
    if (role == kPairSecond) {
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at.val.programmaticStreamSerializationAllowed = 1;
        lc.attrs = &at;
        lc.numAttrs = 1;
    }
    return cudaLaunchKernelEx(&lc, k_walk<BLOCK, ANY, QUANT, Policy>, s, P, n_static, counter, err, depth, knobs | role << 16);
}

// One launch of k_walk, or one of a pair (of which the first may be given a share of the
// GPU only). Stack words: a closest-hit ray leaves one child a level waiting, an any-hit
// ray up to three slots or one word (four_words), a ray of the 8-wide form two
// words a level; the end marker; and the word above the top, which a push writes whether
// it keeps it or not.
template <bool ANY, bool QUANT = false, class Policy>
static cudaError_t launch_walk(const SceneView& s, const Policy& P, uint32_t n_static, uint32_t* counter, uint32_t* err,
                               cudaStream_t stream, const LaunchConfig& cfg, int role = kAlone, int share = 1) {
    int depth = (int)s.depth + 2;
    LaunchConfig c = cfg;
    if (QUANT) {
        depth = 2 * (int)s.wide_depth + 2;
    } else if (ANY) {
        depth = four_words((int)s.depth4);
    }
    // any-hit rays of one origin's neighbourhood profit more from starting together (they
    // read the same nodes; the L1 binds this walk): 16 -> 24 idle lanes, 0.81 -> 0.73 ms
    // for the 5.1M any-hit rays of the 1080p frame. launch_knobs limits it to 32.
    if (ANY) c.refill_min = cfg.refill_min + cfg.refill_min / 2;
    const int knobs = launch_knobs(c);
    switch (cfg.block) {
        case 64: return launch_walk_block<64, ANY, QUANT>(s, P, n_static, counter, err, depth, knobs, role, share, stream);
        case 256: return launch_walk_block<256, ANY, QUANT>(s, P, n_static, counter, err, depth, knobs, role, share, stream);
        default: return launch_walk_block<128, ANY, QUANT>(s, P, n_static, counter, err, depth, knobs, role, share, stream);
    }
}

// launch_walk for the form cfg asks for (has_walk).
template <bool ANY, class Policy>
static cudaError_t launch_rays(const SceneView& s, const Policy& P, uint32_t n_static, uint32_t* counter, uint32_t* err,
                               cudaStream_t stream, const LaunchConfig& cfg, int role = kAlone, int share = 1) {
    return cfg.wide ? launch_walk<ANY, true>(s, P, n_static, counter, err, stream, cfg, role, share)
                    : launch_walk<ANY, false>(s, P, n_static, counter, err, stream, cfg, role, share);
}

}  // namespace timrt
