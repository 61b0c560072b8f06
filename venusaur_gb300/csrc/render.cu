// render.cu -- the plain single-scene wavefront renderer.
//
// Replaces Renderer::Draw (Core/Renderer.h:35-78) and the OptiX programs of
// Core/RayTracer.cu.  A render call is cut into waves of up to max_paths
// paths (pixels x a run of consecutive samples).  Per wave:
//   raygen     one thread per pixel, the wave's samples in order;
//   bounce b   traverse (closest hit for every queued ray)
//              shade    (scatter; survivors compacted into the next queue
//                        with __ballot_sync + a warp prefix, finished paths
//                        write their radiance to their sample slot);
//   accumulate one thread per pixel, Kahan-adds the wave's samples in
//              sample order; the last wave's also writes the running mean
//              (RGBA32F) and sRGB RGBA8.
// Queue counts live on the device; the host never waits inside a render.
#include "render_kernels.cuh"
#include "venu_internal.h"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

namespace venu {

// The bounce loop of a wave (fused variants), run as one CUDA graph or launched
// from the host: the first bounce's kernel, then bounce kernels (odd: queue
// 1 -> 0, even: queue 0 -> 1) while a bounce leaves more rays than the
// finishing kernel takes, then that kernel, which runs the rest of the wave's
// paths to their ends.  In the graph the bounces after the first are a while
// node over a body of two.  The last block of each bounce launch advances the
// loop: it clears the counters the next bounce writes to, counts the bounce,
// and either keeps the loop going or hands what is left to the finishing
// kernel; bounce launches that find no more rays than that do nothing.
struct WaveCtl {
    uint32_t b;            // bounces of the wave traced so far
    uint32_t nb;           // at most this many (the maximum depth)
    uint32_t blocks_done;  // blocks of the running bounce launch that finished
    uint32_t left;         // rays left to the finishing kernel ...
    uint32_t left_q;       // ... in this queue ...
    uint32_t left_first;   // ... or still to be made from the path seeds
    uint32_t left_work;    // hand-out counter of the finishing kernel
    uint32_t pad;
};

// Camera rays of one wave (P pixels from p0, k samples from s0): path
// pos = s * P + pl.  With path_seeds, only each path's raygen seed is written
// (4 bytes instead of a 48-byte queue entry) and the fused kernel makes the
// camera ray itself (PrimaryGen); the pixel's seed still advances through
// every sample's draws, which is what fixes the next sample's seed.
__global__ void k_raygen(venu_camera cam, uint32_t W, uint32_t H, uint32_t p0, uint32_t P, uint32_t s0,
                         uint32_t k, uint32_t subframe, int max_depth, uint32_t* __restrict__ seeds,
                         Queue q, uint32_t* __restrict__ path_seeds, uint32_t* __restrict__ cnt,
                         uint32_t* __restrict__ work, int nbounce, WaveCtl* __restrict__ ctl, uint32_t finish_max,
                         unsigned long long* __restrict__ stats) {
    const uint32_t pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl == 0) {
        cnt[0] = P * k;
        for (int b = 1; b <= nbounce; ++b) cnt[b] = 0;
        for (int b = 0; b <= nbounce; ++b) work[b] = 0;
        if (s0 == 0 && p0 == 0)  // the render's first wave
            for (int i = 0; i < 6; ++i) stats[i] = 0ull;
        ctl->b = 0u;
        ctl->nb = (uint32_t)nbounce;
        ctl->left = P * k <= finish_max ? P * k : 0u;  // a small wave is all the finishing kernel's
        ctl->left_q = 0u;
        ctl->left_first = 1u;
        ctl->left_work = 0u;
    }
    if (pl >= P) return;
    const DevCamera C = load_camera(cam);
    const uint32_t pix = p0 + pl;
    const uint32_t x = pix % W, y = pix / W;
    uint32_t seed = (s0 == 0) ? tea4(pix, subframe) : seeds[pix];
    for (uint32_t s = 0; s < k; ++s) {
        const uint32_t pos = s * P + pl;
        if (path_seeds) path_seeds[pos] = seed;
        f3 o, d;
        camera_ray(C, x, y, W, H, seed, o, d);
        if (!path_seeds) write_primary(q, pos, o, d, pos, max_depth - 1, seed);
    }
    seeds[pix] = seed;
}

// The separate traversal.  WIDE: over the 4-wide tree (variant 5's later
// bounces).  The separate traversal and shading kernels read each queue entry
// and hit record once: they load and store them evict-first
// (ld/st.global.cs), which leaves more of L1 and L2 to the node set (1M
// spheres, variant 3: +0.5 %).  The fused kernel keeps plain accesses: the
// same hints measured -0.45 % on the RTIOW scene there.
//
// A bounce of at least walk_min rays is split over two kernels: this one only
// tests each ray against the sphere it leaves and the hoisted ones, a whole
// warp at a time, and leaves its closest hit so far in the hit record; k_walk
// walks the tree from there with lanes that take a new ray when theirs is
// done.  On large scenes a warp has 12 of 32 lanes in its walk on average
// (its rays take 20 to 400 steps) and waits for L2 most of the time; the
// refills bring that to 24 (10 per instruction: in most steps one or two of them
// test a leaf's sphere while the others wait).  They only pay because a refill is cheap -- the
// up-front tests with their long refined branch are done -- and because lanes
// vote every kWalkSteps steps only and walk on by themselves in between (a
// vote a step costs more than the lanes it fills).  Then the L1 data pipe is
// the bound (85 % of its wavefronts: two 32-byte loads a step and lane).
// Bounces of few rays end with their longest walk either way.
constexpr int32_t kHitDone = 0x40000000;  // in a hit record: nothing left to walk
constexpr int32_t kMissDone = kHitDone | 0x3fffffff;
constexpr int kWalkSteps = 16;
constexpr uint32_t kWalkRefill = 8;  // idle lanes of a warp that fetch together

template <bool COUNT, bool WIDE = false>
__global__ void __launch_bounds__(256) k_traverse(SceneView S, Queue q, const uint32_t* __restrict__ cnt,
                                                  uint32_t* __restrict__ work, int2* __restrict__ hits,
                                                  uint32_t* __restrict__ err,
                                                  unsigned long long* __restrict__ stats, uint32_t walk_min,
                                                  uint32_t leave_max) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    const uint32_t n = *cnt;
    if (n <= leave_max) return;  // the finishing kernel's
    const uint32_t lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats, (unsigned long long)n);
    TraceCounters K{0, 0};
    bool overflow = false;
    if (!COUNT && !WIDE && n >= walk_min) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
            const float4 o4 = __ldcs(q.o + i), d4 = __ldcs(q.d + i);
            RayPre R = prep_for<false>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            float t;
            int32_t k;
            if (!(R.m <= kFarMarginMax)) {  // rare: traced to the end now
                R = prep<false>(R.o, R.d);
                R.from = packed_from(d4.w);
                axis_margins(R);
                k = trace_with<Tracer<false, true, true>>(S, R, 0.0f, 0.001f, 1e16f, t, sm, threadIdx.x, blockDim.x,
                                                          overflow, K);
                k = k < 0 ? kMissDone : k | kHitDone;
            } else {
                Tracer<false> T;
                T.open(R, 0.0f, 0.001f, 1e16f, 1e16f, kNone);
                up_front(T, S, K);
                k = T.result(t);
            }
            hits[i] = make_int2(__float_as_int(t), k);
        }
        if (overflow) atomicOr(err, 1u);
        return;
    }
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(work, 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        const uint32_t i = base + lane;
        if (i < n) {
            float4 o4 = __ldcs(q.o + i), d4 = __ldcs(q.d + i);
            RayPre R = prep_for<COUNT, WIDE>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            float t;
            int32_t k = trace_closest<COUNT, kShared, WIDE>(S, R, 0.001f, 1e16f, t, sm, threadIdx.x, blockDim.x,
                                                           overflow, K);
            __stcs(hits + i, make_int2(__float_as_int(t), k));
        }
    }
    if (overflow) atomicOr(err, 1u);
    if (COUNT) flush_counters(K, stats);
}

__global__ void VENU_WALK_BOUNDS k_walk(SceneView S, Queue q, const uint32_t* __restrict__ cnt,
                                         uint32_t* __restrict__ work, int2* __restrict__ hits,
                                         uint32_t* __restrict__ err, uint32_t walk_min, uint32_t leave_max) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    const uint32_t n = *cnt;
    if (n < walk_min || n <= leave_max) return;  // k_traverse did it, or k_finish will
    const uint32_t lane = threadIdx.x & 31;
    TraceCounters K{0, 0};
    bool overflow = false;
    Tracer<false> T;
    int2 spill[kSpill];
    uint32_t ray = 0;
    bool active = false;
    for (uint32_t idle = 0xffffffffu;;) {
        // the idle lanes take the next rays
        const uint32_t take = (uint32_t)__popc(idle);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(work, take);
        base = __shfl_sync(0xffffffffu, base, 0);
        const bool exhausted = base >= n || n - base <= take;
        if (!active && base < n) {
            ray = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
            if (ray < n) {
                const int2 h = hits[ray];
                if (h.y >= kHitDone) {
                    hits[ray].y = h.y == kMissDone ? -1 : h.y & (kHitDone - 1);
                } else {
                    const float4 o4 = __ldcs(q.o + ray), d4 = __ldcs(q.d + ray);
                    RayPre R = prep_for<false>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
                    R.from = packed_from(d4.w);
                    T.open(R, R.m, 0.001f, 1e16f, __int_as_float(h.x), h.y < 0 ? kNone : h.y);
                    active = T.enter(S, K);  // else the record stands as it is
                }
            }
        }
        // walk until enough lanes are idle, at the end until all are
        const uint32_t enough = exhausted ? 32u : kWalkRefill;
        for (;;) {
            idle = __ballot_sync(0xffffffffu, !active);
            if ((uint32_t)__popc(idle) >= enough) break;
            if (active) {
                for (int i = 0; i < kWalkSteps && active; ++i)
                    active = T.step(S, sm, threadIdx.x, blockDim.x, spill, overflow, K);
                if (!active) {
                    float t;
                    const int32_t k = T.result(t);
                    __stcs(hits + ray, make_int2(__float_as_int(t), k));
                }
            }
        }
        if (exhausted) break;
    }
    if (overflow) atomicOr(err, 1u);
}

// Persistent lanes: a lane whose ray is finished takes a new one as soon as
// at least `refill_min` lanes of its warp are idle (one atomic per refill),
// so warps stay full while the queue lasts instead of waiting for their
// slowest ray (dynamic fetch, Aila & Laine 2009).
template <bool COUNT>
__global__ void __launch_bounds__(256) k_traverse_dyn(SceneView S, Queue q, const uint32_t* __restrict__ cnt,
                                                      uint32_t* __restrict__ work, int2* __restrict__ hits,
                                                      uint32_t* __restrict__ err,
                                                      unsigned long long* __restrict__ stats, uint32_t refill_min) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    const uint32_t n = *cnt;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats, (unsigned long long)n);
    TraceCounters K{0, 0};
    bool overflow = false;
    Tracer<COUNT> T;
    int2 spill[kSpill];
    uint32_t ray = 0;
    bool active = false, exhausted = false;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && (idle == 0xffffffffu || (uint32_t)__popc(idle) >= refill_min)) {
            const uint32_t k = (uint32_t)__popc(idle);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, k);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + k >= n) exhausted = true;
            if (!active) {
                const uint32_t my = base + (uint32_t)__popc(idle & lt);
                if (my < n) {
                    ray = my;
                    const float4 o4 = __ldcs(q.o + my), d4 = __ldcs(q.d + my);
                    RayPre R = prep_for<COUNT>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
                    R.from = packed_from(d4.w);
                    const float m = R.m;  // 0 in counting builds
                    if (COUNT ? R.axis : !(m <= kFarMarginMax)) {
                        // a ray that needs per-axis margins (rare): traced to the
                        // end now with the canonical loop, on this lane's free
                        // stack; the lane stays idle
                        R = prep<false>(R.o, R.d);
                        R.from = packed_from(d4.w);
                        axis_margins(R);
                        float t;
                        const int32_t kk = trace_with<Tracer<COUNT, true, true>>(
                            S, R, 0.0f, 0.001f, 1e16f, t, sm, threadIdx.x, blockDim.x, overflow, K);
                        __stcs(hits + my, make_int2(__float_as_int(t), kk));
                    } else if (T.begin(S, R, m, 0.001f, 1e16f, K)) {
                        active = true;
                    } else {
                        float t;
                        const int32_t kk = T.result(t);
                        __stcs(hits + my, make_int2(__float_as_int(t), kk));
                    }
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (exhausted) break;
            continue;
        }
        if (active && !T.step(S, sm, threadIdx.x, blockDim.x, spill, overflow, K)) {
            active = false;
            float t;
            const int32_t kk = T.result(t);
            __stcs(hits + ray, make_int2(__float_as_int(t), kk));
        }
    }
    if (overflow) atomicOr(err, 1u);
    if (COUNT) flush_counters(K, stats);
}

// One warp-batch loop of the fused kernel: each warp takes 32 rays, traces
// and shades them, and appends the continuing paths to the next queue.
template <bool COUNT, int KS, bool WIDE>
__device__ __forceinline__ void trace_shade_loop(const SceneView& S, const Queue& qin, uint32_t n,
                                                 uint32_t* __restrict__ work, const Queue& qout,
                                                 uint32_t* __restrict__ cnt_out, float4* __restrict__ slots,
                                                 const PrimaryGen& gen, const DevCamera& cam, StackSmem sm,
                                                 bool& overflow, TraceCounters& K) {
    const uint32_t lane = threadIdx.x & 31;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(work, 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        const uint32_t i = base + lane;
        const bool valid = i < n;
        ShadeOut r;
        r.cont = false;
        uint32_t slot = 0;
        if (valid) {
            float4 o4, d4;
            uint32_t seed = 0;
            if (gen.path_seeds) {
                gen_primary(gen, cam, i, o4, d4, seed);
            } else {
                o4 = qin.o[i];
                d4 = qin.d[i];
            }
            slot = (uint32_t)__float_as_int(o4.w);
            RayPre R = prep_for<COUNT, WIDE>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            float t;
            const int32_t k =
                trace_closest<COUNT, KS, WIDE>(S, R, 0.001f, 1e16f, t, sm, threadIdx.x, blockDim.x, overflow, K);
            const float4 t4 = gen.path_seeds ? make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(seed)) : qin.t[i];
            r = shade_one<true>(S, o4, d4, t4, make_int2(__float_as_int(t), k));
        }
        const uint32_t pos = warp_append(r.cont, cnt_out);
        if (r.cont) {
            qout.o[pos] = r.o;
            qout.d[pos] = r.d;
            qout.t[pos] = r.t;
        } else if (valid) {
            slots[slot] = r.result;
        }
    }
}

// The in-place launch (no more rays than the grid has threads): the blocks
// take equal shares of the rays and finish them bounce by bounce.  After
// bounces 1, 2, 4, 8, ... a block brings its surviving paths together (their
// state staged through the unused output queue, at the block's own
// positions); in between each warp runs at its own pace.  This launch waits
// for its longest path (28-31 % of the issue slots used), so a barrier at
// every bounce cost more than the fuller warps gave: against that, 256x144 x 4
// RTIOW 319 -> 303 us, 400x225 x 16 692 -> 679 us; after every 4th or 8th
// bounce only, 400x225 x 16 takes 804 and 1073 us.
// While many paths live they are packed into few warps (issue is what they
// share); from bounce 8 on they are dealt out to all warps of the block, as a
// path runs faster the fewer others its warp takes with it: 256x144 x 4
// 298 -> 275 us, 400x225 x 16 675 -> 651, 300k spheres 512x512 x 4 6.97 ->
// 6.76 ms (from bounce 2: 290 / 666 / 6.74, from 16: 287 / 649 / 6.87).
// Equal shares instead of full blocks first: 64x36 x 2 139 -> 107 us.
// Each path goes through exactly the same arithmetic as in the ordinary loop;
// only the thread that runs it changes.
constexpr uint32_t kSpreadAfter = 8;
template <bool COUNT, int KS, bool WIDE>
__device__ __forceinline__ void trace_shade_in_place(const SceneView& S, const Queue& qin, uint32_t n,
                                                     const Queue& qout, float4* __restrict__ slots,
                                                     bool primary, const PrimaryGen& gen, const DevCamera& cam,
                                                     StackSmem sm, bool& overflow, TraceCounters& K, uint32_t& extra) {
    __shared__ uint32_t warp_live[32];
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5;
    const uint32_t nw = blockDim.x >> 5;
    const uint32_t per = (n + gridDim.x - 1u) / gridDim.x;  // rays of a block
    uint32_t own = t;  // this thread holds the block's own-th state
    const uint32_t base = blockIdx.x * per;
    uint32_t i = base + own;  // this thread's state lives at i
    bool live = own < per && i < n;
    float4 o4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), d4 = o4;
    if (live) {
        uint32_t seed = 0;
        if (primary) {
            gen_primary(gen, cam, i, o4, d4, seed);
            qout.t[i] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(seed));
        } else {
            o4 = qin.o[i];
            d4 = qin.d[i];
            qout.t[i] = qin.t[i];
        }
    }
    uint32_t held = (uint32_t)__syncthreads_count(live);  // threads holding a state, from thread 0 on
    uint32_t done = 0;                                    // bounces traced in place
    for (;;) {
        const uint32_t cnt = (uint32_t)__syncthreads_count(live);
        if (cnt == 0) break;
        const bool spread = done >= kSpreadAfter;
        if (spread ? cnt < held : (cnt + 31u) / 32u < (held + 31u) / 32u) {
            // the live states become the block's states [0, cnt)
            const uint32_t m = __ballot_sync(0xffffffffu, live);
            if (lane == 0) warp_live[w] = (uint32_t)__popc(m);
            float4 t4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (live) t4 = qout.t[i];
            __syncthreads();
            uint32_t pos = (uint32_t)__popc(m & ((1u << lane) - 1u));
            for (uint32_t v = 0; v < w; ++v) pos += warp_live[v];
            if (live) {
                qout.o[base + pos] = o4;
                qout.d[base + pos] = d4;
                qout.t[base + pos] = t4;
            }
            __syncthreads();
            own = spread ? lane * nw + w : t;  // one to each warp in turn
            i = base + own;
            live = own < cnt;
            if (live) {
                o4 = qout.o[i];
                d4 = qout.d[i];
            }
            held = cnt;
        }
        // as many bounces as were traced before, by each warp at its own pace
        const uint32_t until = done ? 2u * done : 1u;
        for (; done < until && __any_sync(0xffffffffu, live); ++done) {
            if (!live) continue;
            RayPre R = prep_for<COUNT, WIDE>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            float th;
            const int32_t k = trace_closest<COUNT, KS, WIDE>(S, R, 0.001f, 1e16f, th, sm, t, blockDim.x, overflow, K);
            const ShadeOut r = shade_one<true>(S, o4, d4, qout.t[i], make_int2(__float_as_int(th), k));
            if (done) ++extra;
            if (r.cont) {
                o4 = r.o;
                d4 = r.d;
                qout.t[i] = r.t;
            } else {
                slots[(uint32_t)__float_as_int(o4.w)] = r.result;
                live = false;
            }
        }
        done = until;
    }
}

// The in-place launch with refills (its own kernel instantiation, REFILL), for
// up to 16 rays per thread of the grid: it finishes every path it takes bounce
// after bounce instead of appending survivors to the next queue.  A warp takes fresh rays
// from the launch (one atomic) between bounces as soon as kRefillLanes of its
// lanes are idle, so its lanes stay busy while paths end at different
// bounces; warps do not wait for one another.  Each path goes through exactly
// the same arithmetic as in the ordinary loop; only the thread that runs it
// changes.  A lane's throughput and seed stay at the position of the first ray
// it took, in the unused output queue.
// Against block-wide refills with a barrier a bounce: 400x225 x 16 RTIOW 757 ->
// 744 us over the wide tree, 656 -> 624 over the binary one, 20k spheres
// 256x256 x 8 838 -> 818 us (8 lanes: 747 / 624 / 812; 16: 756 / 634 / 811).

template <bool COUNT, int KS, bool WIDE>
__device__ __forceinline__ void trace_shade_in_place_refill(const SceneView& S, const Queue& qin, uint32_t n,
                                                     uint32_t* __restrict__ work, const Queue& qout,
                                                     float4* __restrict__ slots, bool primary,
                                                     const PrimaryGen& gen, const DevCamera& cam, StackSmem sm,
                                                     bool& overflow, TraceCounters& K, uint32_t& extra) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t own = 0xffffffffu;  // the first ray this lane took
    bool exhausted = false, live = false, first = false;
    float4 o4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), d4 = o4;
    for (;;) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !live);
        if (!exhausted && (uint32_t)__popc(idle) >= kRefillLanes) {
            const uint32_t take = (uint32_t)__popc(idle);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(work, take);
            base = __shfl_sync(0xffffffffu, base, 0);
            exhausted = base + take >= n;
            const uint32_t ray = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
            if (!live && ray < n) {
                live = first = true;
                if (own == 0xffffffffu) own = ray;
                if (primary) {
                    uint32_t seed = 0;
                    gen_primary(gen, cam, ray, o4, d4, seed);
                    qout.t[own] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(seed));
                } else {
                    o4 = qin.o[ray];
                    d4 = qin.d[ray];
                    qout.t[own] = qin.t[ray];
                }
            }
        }
        if (!__any_sync(0xffffffffu, live)) break;  // only once the launch has no rays left
        if (live) {
            RayPre R = prep_for<COUNT, WIDE>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            float th;
            const int32_t k = trace_closest<COUNT, KS, WIDE>(S, R, 0.001f, 1e16f, th, sm, threadIdx.x, blockDim.x,
                                                           overflow, K);
            const ShadeOut r = shade_one<true>(S, o4, d4, qout.t[own], make_int2(__float_as_int(th), k));
            if (!first) ++extra;
            first = false;
            if (r.cont) {
                o4 = r.o;
                d4 = r.d;
                qout.t[own] = r.t;
            } else {
                slots[(uint32_t)__float_as_int(o4.w)] = r.result;
                live = false;
            }
        }
    }
}

// The end of a bounce launch (see WaveCtl).  handle: the while node's
// condition, 0 for a launch from the host.
__device__ __forceinline__ void wave_advance(WaveCtl* ctl, uint32_t* cnt_in, uint32_t* work, const uint32_t* cnt_out,
                                             uint32_t out_q, uint32_t next_max, unsigned long long* stats,
                                             cudaGraphConditionalHandle handle) {
    __syncthreads();  // every thread of the block is done
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&ctl->blocks_done, 1u) != gridDim.x - 1u) return;
    // the last block: every ray of this bounce is traced and shaded, and its
    // input counters are read by nobody any more
    __threadfence();
    ctl->blocks_done = 0u;
    *cnt_in = 0u;  // the output count of the next bounce
    *work = 0u;    // the hand-out counter of the bounce after it
    const uint32_t b = ctl->b + 1u;
    ctl->b = b;
    const uint32_t next = *reinterpret_cast<const volatile uint32_t*>(cnt_out);
    const bool more = b < ctl->nb && next > next_max;
    if (!more) {
        ctl->left = next <= next_max ? next : 0u;  // after the last bounce there are none
        ctl->left_q = out_q;
        ctl->left_first = 0u;
    }
    if (handle) {
        atomicAdd(stats + 5, 1ull);  // bounce launches run
        cudaGraphSetConditional(handle, more ? 1u : 0u);
    }
}

// Traverse and shade in one pass: each warp takes 32 rays, traverses them,
// then shades all 32 together once the warp has reconverged and appends the
// continuing paths with one ballot and one atomic.  Saves the hit record
// round trip, the second read of the rays and one launch per bounce.
// A launch with at most finish_max rays leaves them to k_finish, as it leaves
// up to next_max continuing rays.
// WIDE: the 4-wide tree instead of the binary traversal records (variant 4,
// k_trace_shade_wide, with its own register cap).
template <bool COUNT, int KS, bool WIDE>
__device__ __forceinline__ void trace_shade_body(const SceneView& S, const Queue& qin,
                                                 uint32_t* __restrict__ cnt_in, uint32_t* __restrict__ work,
                                                 const Queue& qout, uint32_t* __restrict__ cnt_out,
                                                 float4* __restrict__ slots, uint32_t* __restrict__ err,
                                                 unsigned long long* __restrict__ stats, const PrimaryGen& gen,
                                                 WaveCtl* ctl, uint32_t out_q, uint32_t finish_max,
                                                 uint32_t next_max, cudaGraphConditionalHandle handle) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    __shared__ DevCamera cam;  // the primary rays' camera basis, once per block
    const uint32_t n = *cnt_in;
    if (n <= finish_max) {
        if (handle && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(handle, 0u);
        return;
    }
    if (gen.path_seeds) {      // a kernel parameter: the same in every thread
        if (threadIdx.x == 0) cam = load_camera(gen.cam);
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats, (unsigned long long)n);
    TraceCounters K{0, 0};
    bool overflow = false;
    trace_shade_loop<COUNT, KS, WIDE>(S, qin, n, work, qout, cnt_out, slots, gen, cam, sm, overflow, K);
    if (overflow) atomicOr(err, 1u);
    if (COUNT) flush_counters(K, stats);
    wave_advance(ctl, cnt_in, work, cnt_out, out_q, next_max, stats, handle);
}

template <bool COUNT, int KS>
__global__ void VENU_TRACE_BOUNDS k_trace_shade(SceneView S, Queue qin, uint32_t* __restrict__ cnt_in,
                                                uint32_t* __restrict__ work, Queue qout,
                                                uint32_t* __restrict__ cnt_out, float4* __restrict__ slots,
                                                uint32_t* __restrict__ err, unsigned long long* __restrict__ stats,
                                                PrimaryGen gen, WaveCtl* ctl, uint32_t out_q, uint32_t finish_max,
                                                uint32_t next_max, cudaGraphConditionalHandle handle) {
    trace_shade_body<COUNT, KS, false>(S, qin, cnt_in, work, qout, cnt_out, slots, err, stats, gen, ctl, out_q,
                                       finish_max, next_max, handle);
}

template <bool COUNT, int KS>
__global__ void VENU_WIDE_BOUNDS k_trace_shade_wide(SceneView S, Queue qin, uint32_t* __restrict__ cnt_in,
                                                    uint32_t* __restrict__ work, Queue qout,
                                                    uint32_t* __restrict__ cnt_out, float4* __restrict__ slots,
                                                    uint32_t* __restrict__ err,
                                                    unsigned long long* __restrict__ stats, PrimaryGen gen,
                                                    WaveCtl* ctl, uint32_t out_q, uint32_t finish_max,
                                                    uint32_t next_max, cudaGraphConditionalHandle handle) {
    trace_shade_body<COUNT, KS, true>(S, qin, cnt_in, work, qout, cnt_out, slots, err, stats, gen, ctl, out_q,
                                      finish_max, next_max, handle);
}

// What the finishing kernels take: what the bounce kernels noted in WaveCtl, or
// (cnt not null) what the separate traversals left, the first bounce b >= 1 of
// at most leave_max rays.
struct LeftOf {
    const uint32_t* cnt;
    uint32_t nb, leave_max;
};
__device__ __forceinline__ void find_left(const WaveCtl* ctl, LeftOf src, uint32_t& n, bool& primary, bool& second) {
    if (!src.cnt) {
        n = ctl->left;
        primary = ctl->left_first != 0u;
        second = ctl->left_q != 0u;
        return;
    }
    n = 0;
    primary = second = false;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t b0 = 1; b0 < src.nb; b0 += 32u) {
        const uint32_t b = b0 + lane;
        const uint32_t c = b < src.nb ? src.cnt[b] : 0xffffffffu;
        const uint32_t m = __ballot_sync(0xffffffffu, c <= src.leave_max);
        if (m) {
            const int first = __ffs(m) - 1;
            n = __shfl_sync(0xffffffffu, c, first);
            second = ((b0 + (uint32_t)first) & 1u) != 0u;
            return;
        }
    }
}

// The finishing kernel: runs the paths that are left of a wave (WaveCtl) to
// their ends.  A kernel of its own, so that the bounce kernels' code and
// registers are not shaped by it (in one kernel with them, changes to this
// part moved the bounce loop by up to 1.5 %): 1080p x 32 RTIOW 14.05 -> 13.95 ms, 256x144 x 4 278 ->
// 260 us, 64x36 x 2 107 -> 90 us.  At 80 / 96 / 128 registers, with as many
// fewer rays to take, the 256x144 frame takes 297 / 296 / 295 us.  REFILL:
// with refills, for more than spread_max rays (a thread each of the grid); the
// other instantiation takes no more than that.  WIDE: counting builds of variant 4
// alone.  The others finish over the binary tree after either bounce kernel: a
// warp with few active lanes waits for every instruction of a wide step (RTIOW
// 400x225 x 16 654 -> 579 us with variant 4, 256x144 x 4 250 -> 227, 5k random
// spheres 640x360 x 4 655 -> 593, 1280x720 x 8 3.74 -> 3.69 ms).
template <bool COUNT, int KS, bool WIDE, bool REFILL>
__global__ void VENU_FINISH_BOUNDS k_finish(SceneView S, Queue q0, Queue q1, float4* __restrict__ slots,
                                           uint32_t* __restrict__ err, unsigned long long* __restrict__ stats,
                                           PrimaryGen gen, WaveCtl* ctl, uint32_t spread_max, LeftOf src) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    __shared__ DevCamera cam;
    uint32_t n;
    bool primary, second;
    find_left(ctl, src, n, primary, second);
    if (n == 0 || (n > spread_max) != REFILL) return;
    const Queue qin = second ? q1 : q0, qout = second ? q0 : q1;
    if (primary) {
        if (threadIdx.x == 0) cam = load_camera(gen.cam);
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats, (unsigned long long)n);
    TraceCounters K{0, 0};
    bool overflow = false;
    uint32_t extra = 0;  // segments traced after a ray's first
    if (REFILL)
        trace_shade_in_place_refill<COUNT, KS, WIDE>(S, qin, n, &ctl->left_work, qout, slots, primary, gen, cam, sm,
                                                     overflow, K, extra);
    else
        trace_shade_in_place<COUNT, KS, WIDE>(S, qin, n, qout, slots, primary, gen, cam, sm, overflow, K, extra);
    extra = __reduce_add_sync(0xffffffffu, extra);
    if ((threadIdx.x & 31u) == 0 && extra) atomicAdd(stats, (unsigned long long)extra);
    if (overflow) atomicOr(err, 1u);
    if (COUNT) flush_counters(K, stats);
}

// k_finish for large scenes, whose walks are long and uneven (20 to 400 steps): a
// lane whose walk is done does not wait for the other 31.  Once half of a
// warp's paths are through their walks, those are shaded together, start their
// next segments (or new paths) and walk on; the lanes vote every kWalkSteps
// steps, as in k_walk.  Shading and the up-front tests then run for half a warp
// at a time, which long walks pay for and short ones do not.
// Against k_finish, from 7168 spheres up (ms): 8k spheres 1080p x 8 8.28 -> 8.13,
// 100k 1080p x 1 4.37 -> 3.95, 300k 512x512 x 4 with its build 5.72 -> 5.28, 1M
// 1080p x 1 20.8 -> 18.6; 5k 640x480 x 4 0.780 -> 0.797.  Serving at half of the
// paths (an eighth: 19.0 on the last), votes every 16 steps (8: 28.3, 64: 19.3).
__global__ void VENU_WALK_BOUNDS k_finish_walk(SceneView S, Queue q0, Queue q1, float4* __restrict__ slots,
                                               uint32_t* __restrict__ err, unsigned long long* __restrict__ stats,
                                               PrimaryGen gen, WaveCtl* ctl, uint32_t spread_max, LeftOf src) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    __shared__ DevCamera cam;
    uint32_t n;
    bool primary, second;
    find_left(ctl, src, n, primary, second);
    if (n == 0 || n <= spread_max) return;
    const Queue qin = second ? q1 : q0, qout = second ? q0 : q1;
    if (primary) {
        if (threadIdx.x == 0) cam = load_camera(gen.cam);
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u;
    TraceCounters K{0, 0};
    bool overflow = false;
    Tracer<false> T;
    int2 spill[kSpill];
    uint32_t own = 0xffffffffu;  // the first ray this lane took
    uint32_t traced = 0, slot = 0, dbits = 0;
    bool has = false, walking = false, exhausted = false;
    for (;;) {
        float4 o4, d4;
        bool start = false;
        if (has && !walking) {
            float t;
            const int32_t k = T.result(t);
            const ShadeOut r = shade_one<true>(
                S, make_float4(T.R.o.x, T.R.o.y, T.R.o.z, __int_as_float((int)slot)),
                make_float4(T.R.d.x, T.R.d.y, T.R.d.z, __uint_as_float(dbits)), qout.t[own], make_int2(__float_as_int(t), k));
            if (r.cont) {
                o4 = r.o;
                d4 = r.d;
                qout.t[own] = r.t;
                start = true;
            } else {
                slots[slot] = r.result;
                has = false;
            }
        }
        if (!exhausted) {
            const uint32_t empty = __ballot_sync(0xffffffffu, !has);
            const uint32_t take = (uint32_t)__popc(empty);
            if (take) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(&ctl->left_work, take);
                base = __shfl_sync(0xffffffffu, base, 0);
                exhausted = base >= n || n - base <= take;
                const uint32_t ray = base + (uint32_t)__popc(empty & ((1u << lane) - 1u));
                if (!has && base < n && ray < n) {
                    has = start = true;
                    if (own == 0xffffffffu) own = ray;
                    if (primary) {
                        uint32_t seed = 0;
                        gen_primary(gen, cam, ray, o4, d4, seed);
                        qout.t[own] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(seed));
                    } else {
                        o4 = qin.o[ray];
                        d4 = qin.d[ray];
                        qout.t[own] = qin.t[ray];
                    }
                    slot = (uint32_t)__float_as_int(o4.w);
                }
            }
        }
        if (start) {
            ++traced;
            dbits = __float_as_uint(d4.w);
            RayPre R = prep_for<false>(S, mk(o4.x, o4.y, o4.z), mk(d4.x, d4.y, d4.z));
            R.from = packed_from(d4.w);
            const float m = R.m;
            T.open(R, m, 0.001f, 1e16f, 1e16f, kNone);
            if (!(m <= kFarMarginMax)) {  // rare: traced to the end now
                R = prep<false>(R.o, R.d);
                R.from = packed_from(d4.w);
                axis_margins(R);
                float t;
                const int32_t k = trace_with<Tracer<false, true, true>>(S, R, 0.0f, 0.001f, 1e16f, t, sm, threadIdx.x,
                                                                       blockDim.x, overflow, K);
                T.best_t = t;
                T.best = k < 0 ? kNone : k;
            } else {
                up_front(T, S, K);
                walking = T.enter(S, K);
            }
        }
        const uint32_t paths = (uint32_t)__popc(__ballot_sync(0xffffffffu, has));
        if (paths == 0u) break;  // only once there are no rays left
        const uint32_t enough = max(1u, paths >> 1);
        for (;;) {
            const uint32_t w = __ballot_sync(0xffffffffu, walking);
            if (paths - (uint32_t)__popc(w) >= enough) break;
            if (walking)
                for (int i = 0; i < kWalkSteps && walking; ++i)
                    walking = T.step(S, sm, threadIdx.x, blockDim.x, spill, overflow, K);
        }
    }
    traced = __reduce_add_sync(0xffffffffu, traced);
    if (lane == 0 && traced) atomicAdd(stats, (unsigned long long)traced);
    if (overflow) atomicOr(err, 1u);
}

// Separate shading, one ray a thread.  The surviving rays of a block take their
// places in the output queue with one atomic: an atomic a warp came to one a
// nanosecond on the queue's counter (1M spheres 1919x1079 x 8 128.8 -> 127.8 ms;
// caps of 40 and 32 registers 131.6 and 132.9 with an atomic a warp, 128.6 at 40
// with one a block).
__global__ void __launch_bounds__(512) k_shade(SceneView S, Queue qin, const int2* __restrict__ hits,
                                               const uint32_t* __restrict__ cnt_in, Queue qout,
                                               uint32_t* __restrict__ cnt_out, float4* __restrict__ slots,
                                               uint32_t leave_max) {
    const uint32_t n = *cnt_in;
    if (n <= leave_max) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    __shared__ uint32_t found[17];
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t i = base + threadIdx.x;
        ShadeOut r;
        r.cont = false;
        uint32_t slot = 0;
        const bool valid = i < n;
        if (valid) {
            float4 o4 = __ldcs(qin.o + i), d4 = __ldcs(qin.d + i), t4 = __ldcs(qin.t + i);
            slot = (uint32_t)__float_as_int(o4.w);
            r = shade_one<true>(S, o4, d4, t4, __ldcs(hits + i));
        }
        const uint32_t m = __ballot_sync(0xffffffffu, r.cont);
        if (lane == 0) found[warp] = (uint32_t)__popc(m);
        __syncthreads();
        if (warp == 0) {
            const uint32_t mine = lane < warps ? found[lane] : 0u;
            uint32_t sum = mine;
            for (int o = 1; o < 16; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= (uint32_t)o) sum += v;
            }
            uint32_t at = 0;
            if (lane == warps - 1u) at = atomicAdd(cnt_out, sum);
            at = __shfl_sync(0xffffffffu, at, (int)warps - 1);
            if (lane < warps) found[lane] = at + sum - mine;
        }
        __syncthreads();
        const uint32_t pos = found[warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (r.cont) {
            __stcs(qout.o + pos, r.o);
            __stcs(qout.d + pos, r.d);
            __stcs(qout.t + pos, r.t);
        } else if (valid) {
            __stcs(slots + slot, r.result);
        }
    }
}

// Kahan-adds samples [0, k) of pixels [p0, p0+P) from their slots, in order.
// HBM traffic is all it costs, so a render's first wave starts from zero
// (reset) instead of reading a cleared accumulator back, and its last one
// resolves the pixel (the running mean, RGBA32F and sRGB RGBA8) while it holds
// the sums, in place of a clear and a resolve launch.
__global__ void k_accumulate(const float4* __restrict__ slots, uint32_t p0, uint32_t P, uint32_t k,
                             float4* __restrict__ accum, bool reset, float4* __restrict__ image_f,
                             uchar4* __restrict__ image8) {
    const uint32_t pl = blockIdx.x * blockDim.x + threadIdx.x;
    if (pl >= P) return;
    const uint32_t pix = p0 + pl;
    float4 a0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), a1 = a0;
    if (!reset) {
        a0 = accum[2 * (size_t)pix];
        a1 = accum[2 * (size_t)pix + 1];
    }
    for (uint32_t s = 0; s < k; ++s) kahan_add(a0, a1, __ldcs(slots + (size_t)s * P + pl));
    accum[2 * (size_t)pix] = a0;
    accum[2 * (size_t)pix + 1] = a1;
    if (image_f || image8) {
        const f3 mean = mk(a0.x / a0.w, a0.y / a0.w, a0.z / a0.w);
        if (image_f) image_f[pix] = make_float4(mean.x, mean.y, mean.z, 1.0f);
        if (image8) image8[pix] = make_color(mean);
    }
}

__device__ __forceinline__ void load_ray(const float* __restrict__ rays, uint32_t i, f3& o, f3& d) {
    const float* r = rays + 6 * (size_t)i;
    o = mk(r[0], r[1], r[2]);
    d = mk(r[3], r[4], r[5]);
}

// The caller's record of ray i: slot k at distance t, or a miss (k < 0).
__device__ __forceinline__ void store_trace(const SceneView& S, f3 o, f3 d, uint32_t i, float t, int32_t k,
                                            float* __restrict__ t_out, int32_t* __restrict__ id_out,
                                            uint32_t* __restrict__ front_out) {
    if (t_out) t_out[i] = t;
    uint32_t front = 0;
    int32_t id = -1;
    if (k >= 0) {
        id = (int32_t)(__ldg(S.meta + k) & 0x3fffffffu);
        float4 sp = __ldg(S.sph + k);
        f3 p = o + d * t;
        f3 outward = divs(p - mk(sp.x, sp.y, sp.z), sp.w);
        front = dot(d, outward) < 0.0f ? 1u : 0u;
    }
    if (id_out) id_out[i] = id;
    if (front_out) front_out[i] = front;
}

// Arbitrary rays -> closest hit (t, original id, front face), `per_warp` rays a
// warp: 32, or fewer where there are not enough rays for a warp on every
// scheduler (a warp is as slow as all the different walks of its rays
// together): 1001 rays on 20k spheres 137 -> 105 us the whole call, 10k 138 ->
// 120, 1001 on RTIOW 50 -> 45.
// UP_FRONT: only the up-front tests, the closest hit so far left in t_out and
// id_out (a slot, or kNone) for k_trace_walk.
template <bool UP_FRONT>
__global__ void __launch_bounds__(128) k_trace_rays(SceneView S, const float* __restrict__ rays, uint32_t n,
                                                    uint32_t per_warp, float tmin, float tmax,
                                                    float* __restrict__ t_out, int32_t* __restrict__ id_out,
                                                    uint32_t* __restrict__ front_out, uint32_t* __restrict__ err,
                                                    uint32_t* __restrict__ work) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    const uint32_t gt = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    if (UP_FRONT && gt == 0) *work = 0u;
    const uint32_t i = (gt >> 5) * per_warp + lane;
    if (lane >= per_warp || i >= n) return;
    f3 o, d;
    load_ray(rays, i, o, d);
    RayPre R = prep_for<false>(S, o, d);
    TraceCounters K{0, 0};
    bool overflow = false;
    float t;
    if (UP_FRONT) {
        Tracer<false> T;
        T.open(R, 0.0f, tmin, tmax, tmax, kNone);
        up_front(T, S, K);
        t_out[i] = T.best_t;
        id_out[i] = T.best;
        return;
    }
    const int32_t k = trace_closest<false>(S, R, tmin, tmax, t, sm, threadIdx.x, blockDim.x, overflow, K);
    if (overflow) atomicOr(err, 1u);
    store_trace(S, o, d, i, t, k, t_out, id_out, front_out);
}

// The walks of many rays, as k_walk.
__global__ void __launch_bounds__(128, 8) k_trace_walk(SceneView S, const float* __restrict__ rays, uint32_t n, float tmin,
                                                       float tmax, float* __restrict__ t_out,
                                                       int32_t* __restrict__ id_out, uint32_t* __restrict__ front_out,
                                                       uint32_t* __restrict__ err, uint32_t* __restrict__ work) {
    extern __shared__ unsigned char smem[];
    StackSmem sm;
    sm.e = reinterpret_cast<int2*>(smem);
    const uint32_t lane = threadIdx.x & 31;
    TraceCounters K{0, 0};
    bool overflow = false;
    Tracer<false> T;
    int2 spill[kSpill];
    uint32_t ray = 0;
    bool active = false;
    for (uint32_t idle = 0xffffffffu;;) {
        const uint32_t take = (uint32_t)__popc(idle);
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(work, take);
        base = __shfl_sync(0xffffffffu, base, 0);
        const bool exhausted = base >= n || n - base <= take;
        if (!active && base < n) {
            ray = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
            if (ray < n) {
                f3 o, d;
                load_ray(rays, ray, o, d);
                RayPre R = prep_for<false>(S, o, d);
                const float m = R.m, t0 = t_out[ray];
                const int32_t k0 = id_out[ray];
                float t;
                int32_t k;
                if (!(m <= kFarMarginMax)) {  // rare: traced to the end now, on this lane's free stack
                    R = prep<false>(o, d);
                    axis_margins(R);
                    k = trace_with<Tracer<false, true, true>>(S, R, 0.0f, tmin, tmax, t, sm, threadIdx.x, blockDim.x,
                                                              overflow, K);
                } else {
                    T.open(R, m, tmin, tmax, t0, k0);
                    active = T.enter(S, K);
                    k = T.result(t);
                }
                if (!active) store_trace(S, o, d, ray, t, k, t_out, id_out, front_out);
            }
        }
        const uint32_t enough = exhausted ? 32u : kWalkRefill;
        for (;;) {
            idle = __ballot_sync(0xffffffffu, !active);
            if ((uint32_t)__popc(idle) >= enough) break;
            if (active) {
                for (int i = 0; i < kWalkSteps && active; ++i)
                    active = T.step(S, sm, threadIdx.x, blockDim.x, spill, overflow, K);
                if (!active) {
                    float t;
                    const int32_t k = T.result(t);
                    store_trace(S, T.R.o, T.R.d, ray, t, k, t_out, id_out, front_out);
                }
            }
        }
        if (exhausted) break;
    }
    if (overflow) atomicOr(err, 1u);
}

SceneView view_of(const venu_scene* s) {
    SceneView v;
    v.nodes = s->nodes;
    v.sph = s->sph;
    v.mat = s->mat;
    v.meta = s->meta;
    v.trav = s->trav;
    v.wide = s->wide;
    v.n = s->n;
    v.nhoist = s->nhoist;
    for (int i = 0; i < kMaxHoisted; ++i) v.hoist[i] = s->hoist[i];
    if (s->n == 1) {  // no tree: the only sphere is tested up front
        v.nhoist = 1;
        v.hoist[0] = 0;
    }
    return v;
}

// At most 16 KB (256 threads).  No kernel sets cudaFuncAttributeMaxDynamicSharedMemorySize:
// up to 48 KB needs no attribute, and one that a renderer set would be every other
// renderer's limit too (the attribute is the kernel's on the device), so that setting
// up small blocks made the launches of larger ones fail.
static_assert(256 * kShared * sizeof(int2) <= 32 * 1024, "the stacks fit without the attribute");
size_t traverse_smem(int block, int entries) { return (size_t)block * entries * sizeof(int2); }
size_t traverse_smem(int block) { return traverse_smem(block, kShared); }

}  // namespace venu

using namespace venu;

// Everything the wave graph's kernels take as parameters, and their launch
// shape: the graph is rebuilt when any of it changes (zero-initialised, so
// that whole objects compare with memcmp).
struct WaveGraphKey {
    SceneView S;
    PrimaryGen pg;
    Queue q0, q1;
    uint32_t* cnt;
    uint32_t* work;
    float4* slots;
    uint32_t* err;
    unsigned long long* stats;
    WaveCtl* ctl;
    size_t fsm;
    int grid, block, finish_grid;
    uint32_t first_max, finish_max;
    uint32_t kind;  // bits: 4-wide tree, shallow stack, counting build
};

struct venu_renderer {
    uint32_t Q = 0;     // paths the queues hold now (grown on demand up to Qmax)
    uint32_t Qmax = 0;  // the wave size asked for at creation
    uint32_t flags = 0;
    Queue q[2] = {};
    int2* hits = nullptr;
    float4* slots = nullptr;
    uint32_t* seeds = nullptr;
    uint32_t seeds_cap = 0;
    uint32_t* cnt = nullptr;   // [65]
    uint32_t* work = nullptr;  // [65]
    uint32_t* err = nullptr;
    unsigned long long* stats = nullptr;  // segments, nodes, spheres, lane / warp steps, graph bounces
    venu_tuning tune = {2u, 32u, 128u, 0u, 128u, 0u, 1u};
    int trav_blocks = 0, shade_blocks = 0, fused_blocks = 0, finish_blocks = 0, walk_blocks = 0;
    venu_render_stats last = {};
    uint32_t host_launches = 0;  // kernels the last render launched from the host
    bool graph_off = false;      // the wave graph could not be built: host bounce loops only
    // the wave graph (fused variants): built on first use, kept while its key holds
    WaveCtl* ctl = nullptr;
    cudaStream_t cap = nullptr;
    cudaGraph_t wgraph = nullptr;
    cudaGraphExec_t wexec = nullptr;
    WaveGraphKey wkey;
    // VENU_RENDERER_PROFILE: event pairs around traverse (even) / shade (odd) launches
    std::vector<cudaEvent_t> ev;
    size_t ev_used = 0;
};

namespace {
constexpr uint32_t kMaxDepth = 64;
// Where k_traverse is split (variants 0 and 3; ms without -> with, from 1M rays
// up).  By scene, 1080p x 8: 485 spheres 4.96 -> 5.43, 2k 5.00 -> 5.24, 7k 8.73
// -> 8.79, 20k 14.45 -> 14.01, 100k 33.4 -> 30.7, 300k 60.9 -> 54.0, 1M 153.3 ->
// 133.1 (short walks do not need the refills).  By rays: split from 512k up,
// 640x360 x 4 on 300k spheres takes 8.80 instead of 8.48; from 2M up, 1280x720
// x 8 on 1M spheres 65.1 instead of 64.4.
constexpr uint32_t kWalkSpheres = 16384, kWalkRays = 1u << 20;
constexpr uint32_t kShallowSpheres = 4096;      // kSharedShallow stack entries serve up to here
constexpr uint32_t kFinishWalkSpheres = 7168;  // see k_finish_walk
static_assert(kFinishWalkSpheres > kShallowSpheres, "k_finish_walk has the deep stack alone");
template <typename K>
cudaError_t occupancy_grid(K kernel, int block, size_t smem, uint32_t per_sm_cap, int& grid) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem);
    if (e != cudaSuccess) return e;
    per_sm = std::max(1, per_sm);
    if (per_sm_cap) per_sm = std::min(per_sm, (int)per_sm_cap);
    grid = per_sm * sm_count();
    return cudaSuccess;
}

// The fused kernels' launch shape: one for all instantiations of the bounce
// kernel (the shallow-stack ones need less shared memory; same grid) and one for
// those of the finishing kernel.
template <typename K8, typename K4>
cudaError_t configure_fused(venu_renderer* r, K8 deep, K4 shallow) {
    const venu_tuning& t = r->tune;
    const int tb = (int)t.traverse_block;
    const size_t sm = traverse_smem(tb), ss = traverse_smem(tb, kSharedShallow);
    cudaError_t e = occupancy_grid(deep, tb, sm, t.traverse_blocks_per_sm, r->fused_blocks);
    if (e == cudaSuccess)
        e = occupancy_grid(k_finish<false, kShared, false, false>, tb, sm, t.traverse_blocks_per_sm, r->finish_blocks);
    if (e == cudaSuccess) e = prefer_l1(k_finish_walk, std::max(1, r->finish_blocks / std::max(1, sm_count())), sm);
    const int nsm = std::max(1, sm_count());
    const int pb = std::max(1, r->fused_blocks / nsm), pf = std::max(1, r->finish_blocks / nsm);
    if (e == cudaSuccess) e = prefer_l1(deep, pb, sm);
    if (e == cudaSuccess) e = prefer_l1(shallow, pb, ss);
    if (e == cudaSuccess) e = prefer_l1(k_finish<false, kShared, false, false>, pf, sm);
    if (e == cudaSuccess) e = prefer_l1(k_finish<false, kSharedShallow, false, false>, pf, ss);
    if (e == cudaSuccess) e = prefer_l1(k_finish<false, kShared, false, true>, pf, sm);
    if (e == cudaSuccess) e = prefer_l1(k_finish<false, kSharedShallow, false, true>, pf, ss);
    return e;
}

// Persistent grids: as many resident blocks as fit (or the tuned cap) on every SM.
cudaError_t configure(venu_renderer* r) {
    const venu_tuning& t = r->tune;
    const int tb = (int)t.traverse_block;
    const size_t sm = traverse_smem(tb);
    const int nsm = std::max(1, sm_count());
    cudaError_t e = cudaSuccess;
    if (t.traverse_variant == 4) {  // the fused kernel over the 4-wide tree
        e = configure_fused(r, k_trace_shade_wide<false, kShared>, k_trace_shade_wide<false, kSharedShallow>);
        r->trav_blocks = r->fused_blocks;
    } else if (t.traverse_variant >= 2) {  // the fused kernel: every bounce (2), the primary one (3, 5)
        e = configure_fused(r, k_trace_shade<false, kShared>, k_trace_shade<false, kSharedShallow>);
        r->trav_blocks = r->fused_blocks;
    }
    if (e != cudaSuccess) return e;
    if (t.traverse_variant == 5) {  // later bounces: the separate traversal over the wide tree
        e = occupancy_grid(k_traverse<false, true>, tb, sm, t.traverse_blocks_per_sm, r->trav_blocks);
        if (e == cudaSuccess) e = prefer_l1(k_traverse<false, true>, std::max(1, r->trav_blocks / nsm), sm);
    } else if (t.traverse_variant == 0 || t.traverse_variant == 3) {
        e = occupancy_grid(k_traverse<false>, tb, sm, t.traverse_blocks_per_sm, r->trav_blocks);
        if (e == cudaSuccess) e = prefer_l1(k_traverse<false>, std::max(1, r->trav_blocks / nsm), sm);
        if (e == cudaSuccess) e = occupancy_grid(k_walk, tb, sm, t.traverse_blocks_per_sm, r->walk_blocks);
        if (e == cudaSuccess) e = prefer_l1(k_walk, std::max(1, r->walk_blocks / nsm), sm);
    } else if (t.traverse_variant == 1) {
        e = occupancy_grid(k_traverse_dyn<false>, tb, sm, t.traverse_blocks_per_sm, r->trav_blocks);
        if (e == cudaSuccess) e = prefer_l1(k_traverse_dyn<false>, std::max(1, r->trav_blocks / nsm), sm);
    }
    if (e == cudaSuccess) e = occupancy_grid(k_shade, (int)t.shade_block, 0, t.shade_blocks_per_sm, r->shade_blocks);
    if (e == cudaSuccess) e = prefer_l1(k_shade, std::max(1, r->shade_blocks / nsm), 0);
    return e;
}

// Returns an event pair for the next profiled launch, growing the pool.
cudaError_t next_events(venu_renderer* r, cudaEvent_t& a, cudaEvent_t& b) {
    while (r->ev_used + 2 > r->ev.size()) {
        cudaEvent_t e;
        cudaError_t err = cudaEventCreate(&e);
        if (err != cudaSuccess) return err;
        r->ev.push_back(e);
    }
    a = r->ev[r->ev_used];
    b = r->ev[r->ev_used + 1];
    r->ev_used += 2;
    return cudaSuccess;
}

void free_queues(venu_renderer* r) {
    for (int i = 0; i < 2; ++i) {
        cudaFree(r->q[i].o);
        cudaFree(r->q[i].d);
        cudaFree(r->q[i].t);
        r->q[i] = Queue{};
    }
    cudaFree(r->hits);
    cudaFree(r->slots);
    r->hits = nullptr;
    r->slots = nullptr;
    r->Q = 0;
}

// Path queues for waves of Q paths (96 B + 8 B hit + 16 B slot per path).
cudaError_t alloc_queues(venu_renderer* r, uint32_t Q) {
    free_queues(r);
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
        if (e == cudaSuccess) e = cudaMalloc(&r->q[i].o, sizeof(float4) * (size_t)Q);
        if (e == cudaSuccess) e = cudaMalloc(&r->q[i].d, sizeof(float4) * (size_t)Q);
        if (e == cudaSuccess) e = cudaMalloc(&r->q[i].t, sizeof(float4) * (size_t)Q);
    }
    if (e == cudaSuccess) e = cudaMalloc(&r->hits, sizeof(int2) * (size_t)Q);
    if (e == cudaSuccess) e = cudaMalloc(&r->slots, sizeof(float4) * (size_t)Q);
    if (e != cudaSuccess) {
        free_queues(r);
        return e;
    }
    r->Q = Q;
    return cudaSuccess;
}

void destroy_wave_graph(venu_renderer* r);
constexpr uint32_t kFusedWide = 1u, kFusedShallow = 2u, kFusedCount = 4u;

#define VENU_FUSED_CS(LAUNCH, KERNEL)                            \
    do {                                                         \
        if (kind & kFusedCount) {                                \
            if (kind & kFusedShallow) LAUNCH(KERNEL, true, kSharedShallow);  \
            else LAUNCH(KERNEL, true, kShared);                  \
        } else {                                                 \
            if (kind & kFusedShallow) LAUNCH(KERNEL, false, kSharedShallow); \
            else LAUNCH(KERNEL, false, kShared);                 \
        }                                                        \
    } while (0)

// One bounce of the fused kernel (variant 2, or 4 over the 4-wide tree)
// with the renderer's launch shape, into queue out_q.  h: the wave graph's
// loop condition, or 0 for a launch from the host's bounce loop.
cudaError_t launch_fused(const venu_renderer* r, cudaStream_t st, uint32_t kind, size_t fsm, const SceneView& S,
                         uint32_t* cnt_in, uint32_t* work, uint32_t out_q, uint32_t* cnt_out, const PrimaryGen& pg,
                         uint32_t finish_max, uint32_t next_max, cudaGraphConditionalHandle h) {
    const int grid = r->fused_blocks, tb = (int)r->tune.traverse_block;
    const Queue &qi = r->q[1u - out_q], &qo = r->q[out_q];
#define VENU_FUSED(KERNEL, C, KS)                                                                              \
    KERNEL<C, KS><<<grid, tb, fsm, st>>>(S, qi, cnt_in, work, qo, cnt_out, r->slots, r->err, r->stats, pg, r->ctl, \
                                         out_q, finish_max, next_max, h)
    if (kind & kFusedWide) VENU_FUSED_CS(VENU_FUSED, k_trace_shade_wide);
    else VENU_FUSED_CS(VENU_FUSED, k_trace_shade);
#undef VENU_FUSED
    return cudaGetLastError();
}

// What is left of a wave (see WaveCtl): by the refilling kernel, by the
// spreading one, or by whichever finds its number of rays.
constexpr uint32_t kFinishRefill = 1u, kFinishSpread = 2u;
cudaError_t launch_finish(const venu_renderer* r, cudaStream_t st, uint32_t kind, size_t fsm, const SceneView& S,
                          const PrimaryGen& pg, uint32_t which, LeftOf src = LeftOf{nullptr, 0u, 0u}) {
    const int grid = r->finish_blocks, tb = (int)r->tune.traverse_block;
    const uint32_t spread_max = (uint32_t)grid * (uint32_t)tb;
    const bool walk = S.n >= kFinishWalkSpheres && !(kind & kFusedCount);
#define VENU_FINISH(WIDE, C, KS)                                                                                  \
    do {                                                                                                          \
        if (walk && (which & kFinishRefill))                                                                      \
            k_finish_walk<<<grid, tb, fsm, st>>>(S, r->q[0], r->q[1], r->slots, r->err, r->stats, pg, r->ctl,     \
                                                 spread_max, src);                                                \
        else if (which & kFinishRefill)                                                                           \
            k_finish<C, KS, C && WIDE, true>                                                                           \
                <<<grid, tb, fsm, st>>>(S, r->q[0], r->q[1], r->slots, r->err, r->stats, pg, r->ctl, spread_max, src); \
        if (which & kFinishSpread)                                                                                \
            k_finish<C, KS, C && WIDE, false>                                                                          \
                <<<grid, tb, fsm, st>>>(S, r->q[0], r->q[1], r->slots, r->err, r->stats, pg, r->ctl, spread_max, src); \
    } while (0)
    if (kind & kFusedWide) VENU_FUSED_CS(VENU_FINISH, true);
    else VENU_FUSED_CS(VENU_FINISH, false);
#undef VENU_FINISH
    return cudaGetLastError();
}
#undef VENU_FUSED_CS

// Builds the wave graph for `key` (see WaveCtl): the first bounce (camera
// rays from the per-path seeds, queue 0 -> 1), while (more rays than the
// finishing kernel takes) { queue 1 -> 0; queue 0 -> 1 }, the finishing
// kernel.  After an odd bounce that ends the loop the even one still starts
// and finds nothing to do.
venu_status build_wave_graph(venu_renderer* r, const WaveGraphKey& key) {
    destroy_wave_graph(r);
    if (!r->cap) VENU_CUDA(cudaStreamCreateWithFlags(&r->cap, cudaStreamNonBlocking));
    VENU_CUDA(cudaGraphCreate(&r->wgraph, 0));
    cudaGraph_t g = r->wgraph;
    cudaGraphConditionalHandle h = 0;
    VENU_CUDA(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
    PrimaryGen later = key.pg;
    later.path_seeds = nullptr;  // bounces after the first read their rays from the queue
    VENU_CUDA(cudaStreamBeginCaptureToGraph(r->cap, g, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    cudaError_t le = launch_fused(r, r->cap, key.kind, key.fsm, key.S, key.cnt, key.work, 1u, key.cnt + 1, key.pg,
                                  key.first_max, key.finish_max, h);
    cudaGraph_t captured = nullptr;
    cudaError_t ee = cudaStreamEndCapture(r->cap, &captured);
    if (le != cudaSuccess) return cuda_fail(le, "venu_render: capture of the first bounce");
    if (ee != cudaSuccess) return cuda_fail(ee, "venu_render: cudaStreamEndCapture");
    cudaGraphNode_t first = nullptr;
    size_t nn = 1;
    VENU_CUDA(cudaGraphGetNodes(g, &first, &nn));
    if (nn != 1) {
        set_error("venu_render: the first bounce captured as " + std::to_string(nn) + " graph nodes");
        return VENU_ERR_CUDA;
    }
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t loop = nullptr;
    VENU_CUDA(cudaGraphAddNode(&loop, g, &first, nullptr, 1, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    VENU_CUDA(cudaStreamBeginCaptureToGraph(r->cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
    le = launch_fused(r, r->cap, key.kind, key.fsm, key.S, key.cnt + 1, key.work + 1, 0u, key.cnt, later,
                      key.finish_max, key.finish_max, h);
    if (le == cudaSuccess)
        le = launch_fused(r, r->cap, key.kind, key.fsm, key.S, key.cnt, key.work, 1u, key.cnt + 1, later,
                          key.finish_max, key.finish_max, h);
    ee = cudaStreamEndCapture(r->cap, &captured);
    if (le != cudaSuccess) return cuda_fail(le, "venu_render: capture of the bounce loop");
    if (ee != cudaSuccess) return cuda_fail(ee, "venu_render: cudaStreamEndCapture");
    VENU_CUDA(cudaStreamBeginCaptureToGraph(r->cap, g, &loop, nullptr, 1, cudaStreamCaptureModeRelaxed));
    le = launch_finish(r, r->cap, key.kind, key.fsm, key.S, key.pg, kFinishRefill | kFinishSpread);
    ee = cudaStreamEndCapture(r->cap, &captured);
    if (le != cudaSuccess) return cuda_fail(le, "venu_render: capture of the finishing kernel");
    if (ee != cudaSuccess) return cuda_fail(ee, "venu_render: cudaStreamEndCapture");
    VENU_CUDA(cudaGraphInstantiate(&r->wexec, g, 0));
    r->wkey = key;
    return VENU_OK;
}

void destroy_wave_graph(venu_renderer* r) {
    if (r->wexec) cudaGraphExecDestroy(r->wexec);
    if (r->wgraph) cudaGraphDestroy(r->wgraph);
    r->wexec = nullptr;
    r->wgraph = nullptr;
}

void free_renderer(venu_renderer* r) {
    for (cudaEvent_t e : r->ev) cudaEventDestroy(e);
    r->ev.clear();
    destroy_wave_graph(r);
    if (r->cap) cudaStreamDestroy(r->cap);
    r->cap = nullptr;
    cudaFree(r->ctl);
    free_queues(r);
    cudaFree(r->seeds);
    cudaFree(r->cnt);
    cudaFree(r->work);
    cudaFree(r->err);
    cudaFree(r->stats);
}
}  // namespace

extern "C" venu_status venu_renderer_create(uint32_t max_paths, uint32_t flags, venu_renderer** out) {
    if (!out) {
        set_error("venu_renderer_create: out is NULL");
        return VENU_ERR_INVALID;
    }
    *out = nullptr;
    venu_status ds = require_device();
    if (ds != VENU_OK) return ds;
    if (max_paths == 0) max_paths = 64u << 20;
    // 2^30 keeps every path position and slot below 2^31 (signed slot words,
    // FastDiv's range) at ~120 B per path (~129 GB at the maximum)
    if (max_paths > (1u << 30)) {
        set_error("venu_renderer_create: max_paths above 2^30");
        return VENU_ERR_TOO_LARGE;
    }
    venu_renderer* r = new venu_renderer();
    r->Qmax = max_paths;  // the queues are sized by the first render that needs them
    r->flags = flags;
    cudaError_t e = cudaMalloc(&r->cnt, sizeof(uint32_t) * (kMaxDepth + 1));
    if (e == cudaSuccess) e = cudaMalloc(&r->work, sizeof(uint32_t) * (kMaxDepth + 1));
    if (e == cudaSuccess) e = cudaMalloc(&r->err, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMalloc(&r->stats, sizeof(unsigned long long) * 6);
    if (e == cudaSuccess) e = cudaMemset(r->err, 0, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(r->stats, 0, sizeof(unsigned long long) * 6);
    if (e == cudaSuccess) e = cudaMalloc(&r->ctl, sizeof(WaveCtl));
    if (e == cudaSuccess) e = cudaMemset(r->ctl, 0, sizeof(WaveCtl));
    if (e == cudaSuccess) e = configure(r);
    if (e != cudaSuccess) {
        free_renderer(r);
        delete r;
        return e == cudaErrorMemoryAllocation ? (set_error("venu_renderer_create: out of device memory"), VENU_ERR_OOM)
                                              : cuda_fail(e, "venu_renderer_create");
    }
    *out = r;
    return VENU_OK;
}

extern "C" venu_status venu_renderer_set_tuning(venu_renderer* r, const venu_tuning* t) {
    if (!r || !t) {
        set_error("venu_renderer_set_tuning: NULL argument");
        return VENU_ERR_INVALID;
    }
    const bool ok = t->traverse_variant <= 5u && t->refill_min >= 1u && t->refill_min <= 32u &&
                    (t->traverse_block == 64u || t->traverse_block == 128u || t->traverse_block == 256u) &&
                    t->shade_block >= 64u && t->shade_block <= 512u && (t->shade_block % 32u) == 0u &&
                    t->traverse_blocks_per_sm <= 32u && t->shade_blocks_per_sm <= 32u && t->in_place_factor <= 16u;
    if (!ok) {
        set_error("venu_renderer_set_tuning: value out of range");
        return VENU_ERR_INVALID;
    }
    const venu_tuning old = r->tune;
    r->tune = *t;
    cudaError_t e = configure(r);
    if (e != cudaSuccess) {
        r->tune = old;
        configure(r);
        return cuda_fail(e, "venu_renderer_set_tuning");
    }
    return VENU_OK;
}

extern "C" venu_status venu_renderer_get_tuning(const venu_renderer* r, venu_tuning* t) {
    if (!r || !t) {
        set_error("venu_renderer_get_tuning: NULL argument");
        return VENU_ERR_INVALID;
    }
    *t = r->tune;
    return VENU_OK;
}

extern "C" venu_status venu_renderer_destroy(venu_renderer* r) {
    if (!r) return VENU_OK;
    free_renderer(r);
    delete r;
    return VENU_OK;
}

extern "C" venu_status venu_render(venu_renderer* r, const venu_scene* scene, const venu_camera* camera,
                                   const venu_render_opts* opts, float* accum_dev, float* image_f_dev,
                                   uint8_t* image8_dev, void* stream) {
    if (!r || !scene || !camera || !opts || !accum_dev) {
        set_error("venu_render: NULL argument");
        return VENU_ERR_INVALID;
    }
    const uint32_t W = opts->width, H = opts->height, spp = opts->samples_per_pixel;
    const uint32_t maxd = opts->max_depth;
    if (W < 2 || H < 2 || spp == 0 || maxd == 0 || maxd > kMaxDepth) {
        set_error("venu_render: need width,height >= 2, spp >= 1, 1 <= max_depth <= 64");
        return VENU_ERR_INVALID;
    }
    const uint64_t npix64 = (uint64_t)W * H;
    if (npix64 > (1u << 30)) {
        set_error("venu_render: image above 2^30 pixels");
        return VENU_ERR_TOO_LARGE;
    }
    const uint32_t npix = (uint32_t)npix64;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (npix > r->seeds_cap) {
        cudaFree(r->seeds);
        r->seeds = nullptr;
        r->seeds_cap = 0;
        VENU_CUDA(cudaMalloc(&r->seeds, sizeof(uint32_t) * npix));
        r->seeds_cap = npix;
    }
    const bool reset = (opts->flags & VENU_FLAG_RESET_ACCUM) != 0;
    if (r->tune.traverse_variant == 4u || r->tune.traverse_variant == 5u) {
        const venu_status ws = ensure_wide(scene, st);  // the first such render builds it
        if (ws != VENU_OK) return ws;
    }
    const SceneView S = view_of(scene);
    const bool count = (r->flags & VENU_RENDERER_COUNT) != 0;
    const bool prof = (r->flags & VENU_RENDERER_PROFILE) != 0;
    r->ev_used = 0;
    {
        // queues for waves of min(all paths of this call, Qmax): a small render
        // holds no more memory than it uses; grown (never shrunk) on demand
        const uint64_t want = std::min<uint64_t>((uint64_t)npix * spp, r->Qmax);
        if (want > r->Q) {
            VENU_CUDA(cudaStreamSynchronize(st));
            const cudaError_t ae = alloc_queues(r, (uint32_t)want);
            if (ae != cudaSuccess) {
                set_error("venu_render: cannot allocate path queues for " + std::to_string(want) + " paths");
                return VENU_ERR_OOM;
            }
        }
    }
    const venu_tuning& tu = r->tune;
    const size_t tsm = traverse_smem((int)tu.traverse_block);
    const int tb = (int)tu.traverse_block, sb = (int)tu.shade_block;
    float4* accum = reinterpret_cast<float4*>(accum_dev);
    uint32_t launches = 0, waves = 0;
    // wave shape: all pixels x k samples, or P pixels x 1 sample
    uint32_t P, k;
    if (npix <= r->Q) {
        P = npix;
        k = std::min(spp, r->Q / npix);
    } else {
        P = r->Q;
        k = 1;
    }
    const int nb = (int)maxd;
    // the fused first bounce (variants 2 and 3) makes its camera rays from
    // per-path seeds, kept in the first queue's throughput array (bounce 0
    // reads no queue and writes the other one)
    const bool gen0 = tu.traverse_variant >= 2u;
    // small scenes have shallow trees: a 4-entry shared stack leaves more of
    // the SM's memory to L1 (measured: RTIOW +0.5 %; 1M spheres -4.5 %)
    const bool shallow = scene->n <= kShallowSpheres;
    uint32_t* const path_seeds = gen0 ? reinterpret_cast<uint32_t*>(r->q[0].t) : nullptr;
    // bounces that k_walk takes (see k_traverse): counting builds never split
    const uint32_t walk_min =
        !count && scene->n >= kWalkSpheres && (uint64_t)npix * k >= kWalkRays ? kWalkRays : ~0u;
    // the fused variants run each wave's bounce loop as one graph launch
    // (WaveCtl) when every wave covers all pixels, so that the graph's
    // parameters are the same for every wave; the profiling build times
    // every launch from the host
    const bool fused = tu.traverse_variant == 2u || tu.traverse_variant == 4u;
    // a caller capturing the stream into a graph of its own gets the
    // host's bounce loop captured (no graph launched inside the capture)
    cudaStreamCaptureStatus cap_status = cudaStreamCaptureStatusNone;
    VENU_CUDA(cudaStreamIsCapturing(st, &cap_status));
    bool use_graph = fused && !prof && P == npix && !r->graph_off && cap_status == cudaStreamCaptureStatusNone;
    const uint32_t kind = (tu.traverse_variant == 4u ? kFusedWide : 0u) | (shallow ? kFusedShallow : 0u) |
                          (count ? kFusedCount : 0u);
    const size_t fsm = shallow ? traverse_smem(tb, kSharedShallow) : tsm;
    // the camera-ray generator of the wave of pixels [p0, p0 + PP)
    auto primary_gen = [&](uint32_t p0, uint32_t PP) {
        PrimaryGen pg;
        std::memset(&pg, 0, sizeof pg);  // the graph key compares whole objects
        pg.cam = *camera;
        pg.W = W;
        pg.H = H;
        pg.p0 = p0;
        pg.P = PP;
        pg.depth = (int)maxd - 1;
        pg.div_P = make_fastdiv(PP);
        pg.div_W = make_fastdiv(W);
        return pg;
    };
    // The finishing kernels take whole waves of at most first_max rays and, of the
    // fused variants, what a bounce leaves when that is at most finish_max.  An
    // in_place_factor above 1 asks for that many rays per thread of their grid.
    // Otherwise: up to 16, but whole waves only of small scenes, where camera
    // rays lose little by sharing warps with later bounces; of large ones a ray
    // per thread (ms at 1 / 8 / 16 for both): RTIOW 400x225 x 16 0.625 / 0.572 /
    // 0.558, 1280x720 x 1 at depth 4 0.495 / 0.431 / 0.430, 300k spheres 512x512 x
    // 4 with its build 6.73 / 5.89 / 5.90; but 100k 1080p x 1, whose 2.1M camera
    // rays only 16 takes, 4.99 / 4.46 / 5.16.
    const uint64_t threads = (uint64_t)r->finish_blocks * (uint64_t)tb;
    // Scenes that k_finish_walk serves are its own after the first bounce (at 16 /
    // 64 / any number of rays a thread, 1080p x 8 on 20k spheres takes 12.9 / 12.9 /
    // 12.5 ms, on 300k 54.7 / 52.0 / 50.5; RTIOW at any number 15.0 instead of 13.3
    // over its bounces); after the separate traversals it takes up to 32 (1M 1919x1079
    // x 8 at 8 / 16 / 32 / 64: 131.0 / 129.6 / 129.2 / 130.3 ms).
    const bool walks = scene->n >= kFinishWalkSpheres && !count;
    const uint64_t asked = tu.in_place_factor > 1u ? tu.in_place_factor : !walks ? 16u : fused ? 1u << 20 : 32u;
    const uint32_t finish_max = gen0 ? (uint32_t)std::min<uint64_t>(asked * threads, 0xffffffffu) : 0u;
    const uint32_t first_max =
        gen0 ? (uint32_t)(tu.in_place_factor > 1u || shallow ? finish_max : threads) : 0u;
    const uint32_t bounce_max = fused ? finish_max : 0u;
    const uint32_t leave_max = gen0 && !fused ? finish_max : 0u;
    use_graph = use_graph && (uint64_t)npix * k > first_max;
    if (use_graph) {
        WaveGraphKey key;
        std::memset(&key, 0, sizeof key);
        key.S = S;
        key.pg = primary_gen(0u, npix);
        key.pg.path_seeds = path_seeds;
        key.q0 = r->q[0];
        key.q1 = r->q[1];
        key.cnt = r->cnt;
        key.work = r->work;
        key.slots = r->slots;
        key.err = r->err;
        key.stats = r->stats;
        key.ctl = r->ctl;
        key.fsm = fsm;
        key.grid = r->fused_blocks;
        key.finish_grid = r->finish_blocks;
        key.first_max = first_max;
        key.finish_max = finish_max;
        key.block = tb;
        key.kind = kind;
        if (!r->wexec || std::memcmp(&key, &r->wkey, sizeof key) != 0) {
            if (build_wave_graph(r, key) != VENU_OK) {
                // graphs unavailable here: the host's bounce loop from now on
                destroy_wave_graph(r);
                (void)cudaGetLastError();
                r->graph_off = true;
                use_graph = false;
            }
        }
    }
    for (uint32_t s0 = 0; s0 < spp; s0 += k) {
        const uint32_t kk = std::min(k, spp - s0);
        for (uint32_t p0 = 0; p0 < npix; p0 += P) {
            const uint32_t PP = std::min(P, npix - p0);
            k_raygen<<<(PP + 255) / 256, 256, 0, st>>>(*camera, W, H, p0, PP, s0, kk, opts->subframe_index,
                                                       (int)maxd, r->seeds, r->q[0], path_seeds, r->cnt, r->work,
                                                       nb, r->ctl, first_max, r->stats);
            PrimaryGen pg = primary_gen(p0, PP);
            pg.path_seeds = path_seeds;
            const bool small = (uint64_t)PP * kk <= first_max;
            const uint32_t which = !small                               ? kFinishRefill | kFinishSpread
                                   : (uint64_t)PP * kk > threads ? kFinishRefill
                                                                        : kFinishSpread;
            const uint32_t finishes = small ? 1u : 2u;
            ++launches;
            if (small) {
                if (prof) {
                    for (int i = 0; i < 2; ++i) {
                        cudaEvent_t a, z;
                        VENU_CUDA(next_events(r, a, z));
                        VENU_CUDA(cudaEventRecord(a, st));
                        if (i == 0) VENU_CUDA(launch_finish(r, st, kind, fsm, S, pg, which));
                        VENU_CUDA(cudaEventRecord(z, st));
                    }
                } else {
                    VENU_CUDA(launch_finish(r, st, kind, fsm, S, pg, which));
                }
                launches += finishes;
            } else if (use_graph) {  // the bounce loop of this wave: one graph launch
                VENU_CUDA(cudaGraphLaunch(r->wexec, st));
                launches += finishes;  // the bounces count themselves
            }
            for (int b = 0; b < nb && !small && !use_graph; ++b) {
                const Queue& qi = r->q[b & 1];
                const Queue& qo = r->q[(b + 1) & 1];
                cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr, e3 = nullptr;
                if (prof) {
                    VENU_CUDA(next_events(r, e0, e1));
                    VENU_CUDA(next_events(r, e2, e3));
                    VENU_CUDA(cudaEventRecord(e0, st));
                }
                // variant 3: the coherent primary rays fused, the divergent
                // later bounces with the separate traversal kernel
                const uint32_t v = tu.traverse_variant <= 2u ? tu.traverse_variant
                                   : tu.traverse_variant == 4u ? 4u
                                   : tu.traverse_variant == 5u ? (b == 0 ? 2u : 5u)
                                                               : (b == 0 ? 2u : 0u);
                if ((v == 4 || v == 5) && scene->nwide == 0u && scene->n > 1u) {
                    set_error("venu_render: the scene has no wide tree");
                    return VENU_ERR_INVALID;
                }
                if (v == 2 || v == 4) {
                    pg.path_seeds = (b == 0) ? path_seeds : nullptr;
                    VENU_CUDA(launch_fused(r, st, kind, fsm, S, r->cnt + b, r->work + b, (uint32_t)((b + 1) & 1),
                                           r->cnt + b + 1, pg, b == 0 ? 0u : bounce_max, bounce_max, 0));
                    if (prof) {
                        VENU_CUDA(cudaEventRecord(e1, st));
                        VENU_CUDA(cudaEventRecord(e2, st));
                        VENU_CUDA(cudaEventRecord(e3, st));
                    }
                    launches += 1;
                    continue;
                }
                if (v == 0) {
                    if (count)
                        k_traverse<true><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b, r->hits,
                                                                         r->err, r->stats, ~0u, leave_max);
                    else
                        k_traverse<false><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b, r->hits,
                                                                          r->err, r->stats, walk_min, leave_max);
                    if (walk_min != ~0u) {
                        k_walk<<<r->walk_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b, r->hits, r->err,
                                                                walk_min, leave_max);
                        ++launches;
                    }
                } else if (v == 5) {
                    if (count)
                        k_traverse<true, true><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b,
                                                                               r->hits, r->err, r->stats, ~0u, leave_max);
                    else
                        k_traverse<false, true><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b,
                                                                                r->hits, r->err, r->stats, ~0u, leave_max);
                } else {
                    if (count)
                        k_traverse_dyn<true><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b, r->hits,
                                                                             r->err, r->stats, tu.refill_min);
                    else
                        k_traverse_dyn<false><<<r->trav_blocks, tb, tsm, st>>>(S, qi, r->cnt + b, r->work + b,
                                                                              r->hits, r->err, r->stats, tu.refill_min);
                }
                if (prof) {
                    VENU_CUDA(cudaEventRecord(e1, st));
                    VENU_CUDA(cudaEventRecord(e2, st));
                }
                k_shade<<<r->shade_blocks, sb, 0, st>>>(S, qi, r->hits, r->cnt + b, qo, r->cnt + b + 1, r->slots,
                                                        leave_max);
                if (prof) VENU_CUDA(cudaEventRecord(e3, st));
                launches += 2;
            }
            if (gen0 && !small && !use_graph) {  // what the bounces left
                const LeftOf src = fused ? LeftOf{nullptr, 0u, 0u} : LeftOf{r->cnt, (uint32_t)nb, leave_max};
                if (prof) {
                    for (int i = 0; i < 2; ++i) {
                        cudaEvent_t a, z;
                        VENU_CUDA(next_events(r, a, z));
                        VENU_CUDA(cudaEventRecord(a, st));
                        if (i == 0) VENU_CUDA(launch_finish(r, st, kind, fsm, S, pg, which, src));
                        VENU_CUDA(cudaEventRecord(z, st));
                    }
                } else {
                    VENU_CUDA(launch_finish(r, st, kind, fsm, S, pg, which, src));
                }
                launches += finishes;
            }
            const bool last = s0 + kk == spp;  // of these pixels
            k_accumulate<<<(PP + 255) / 256, 256, 0, st>>>(
                r->slots, p0, PP, kk, accum, reset && s0 == 0, last ? reinterpret_cast<float4*>(image_f_dev) : nullptr,
                last ? reinterpret_cast<uchar4*>(image8_dev) : nullptr);
            ++launches;
            ++waves;
        }
    }
    VENU_CUDA(cudaGetLastError());
    r->last = venu_render_stats{};
    r->last.paths = (uint64_t)npix * spp;
    r->last.waves = waves;
    r->last.kernel_launches = launches;  // plus the wave graphs' bounces, counted on the device
    r->host_launches = launches;
    return VENU_OK;
}

extern "C" venu_status venu_renderer_stats(venu_renderer* r, venu_render_stats* out) {
    if (!r || !out) {
        set_error("venu_renderer_stats: NULL argument");
        return VENU_ERR_INVALID;
    }
    unsigned long long st[6] = {0, 0, 0, 0, 0, 0};
    uint32_t err = 0;
    VENU_CUDA(cudaMemcpy(st, r->stats, sizeof(st), cudaMemcpyDeviceToHost));
    VENU_CUDA(cudaMemcpy(&err, r->err, sizeof(err), cudaMemcpyDeviceToHost));
    r->last.segments = st[0];
    r->last.nodes_visited = st[1];
    r->last.spheres_tested = st[2];
    r->last.lane_steps = st[3];
    r->last.warp_steps = st[4];
    r->last.kernel_launches = r->host_launches + (uint32_t)st[5];
    // event pairs alternate traverse, shade (4 events per bounce)
    float tms = 0.0f, sms = 0.0f;
    uint32_t tn = 0, sn = 0;
    for (size_t i = 0; i + 3 < r->ev_used; i += 4) {
        float a = 0.0f, b = 0.0f;
        VENU_CUDA(cudaEventElapsedTime(&a, r->ev[i], r->ev[i + 1]));
        VENU_CUDA(cudaEventElapsedTime(&b, r->ev[i + 2], r->ev[i + 3]));
        tms += a;
        sms += b;
        ++tn;
        ++sn;
    }
    r->last.traverse_ms = tms;
    r->last.shade_ms = sms;
    r->last.traverse_launches = tn;
    r->last.shade_launches = sn;
    *out = r->last;
    if (err) {
        set_error("traversal stack overflow (result of at least one ray is incomplete)");
        return VENU_ERR_STACK;
    }
    return VENU_OK;
}

extern "C" venu_status venu_trace(const venu_scene* scene, const float* rays_dev, uint32_t n, float tmin,
                                  float tmax, float* t_dev, int32_t* id_dev, uint32_t* front_dev, void* stream) {
    if (!scene || (!rays_dev && n)) {
        set_error("venu_trace: NULL argument");
        return VENU_ERR_INVALID;
    }
    venu_status ds = require_device();
    if (ds != VENU_OK) return ds;
    if (n == 0) return VENU_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // an error word of the scene's (0 unless a call failed), so that a call
    // neither allocates nor clears; one of its own for more calls at once than
    // there are, and for a scene without spheres
    uint32_t* err = nullptr;
    int word = -1;
    if (scene->trace_err) {
        std::lock_guard<std::mutex> lock(scene->trace_mu);
        for (uint32_t i = 0; i < kTraceWords / 2 && word < 0; ++i)
            if (!(scene->trace_used >> i & 1u)) word = (int)i;
        if (word >= 0) scene->trace_used |= 1ull << word;
    }
    cudaError_t e = cudaSuccess;
    if (word >= 0) {
        err = scene->trace_err + 2 * word;
    } else {
        VENU_CUDA(cudaMalloc(&err, 2 * sizeof(uint32_t)));
        e = cudaMemsetAsync(err, 0, 2 * sizeof(uint32_t), st);
    }
    const size_t tsm = traverse_smem((int)kTraceBlock);
    if (e == cudaSuccess) {
        const SceneView S = view_of(scene);
        const TracePlan P = trace_plan(scene->n, n, t_dev && id_dev, (uint32_t)sm_count());
        if (P.walk) {
            k_trace_rays<true><<<P.grid, kTraceBlock, tsm, st>>>(S, rays_dev, n, P.per_warp, tmin, tmax, t_dev, id_dev,
                                                                front_dev, err, err + 1);
            k_trace_walk<<<sm_count() * 8, kTraceBlock, tsm, st>>>(S, rays_dev, n, tmin, tmax, t_dev, id_dev, front_dev,
                                                                 err, err + 1);
        } else {
            k_trace_rays<false><<<P.grid, kTraceBlock, tsm, st>>>(S, rays_dev, n, P.per_warp, tmin, tmax, t_dev, id_dev,
                                                                 front_dev, err, nullptr);
        }
        e = cudaGetLastError();
    }
    uint32_t herr = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (word >= 0) {
        if (herr) {
            cudaMemsetAsync(err, 0, sizeof(uint32_t), st);
            cudaStreamSynchronize(st);
        }
        std::lock_guard<std::mutex> lock(scene->trace_mu);
        scene->trace_used &= ~(1ull << word);
    } else {
        cudaFree(err);
    }
    if (e != cudaSuccess) return cuda_fail(e, "venu_trace");
    if (herr) {
        set_error("venu_trace: traversal stack overflow");
        return VENU_ERR_STACK;
    }
    return VENU_OK;
}
