// lbvh.cu -- linear BVH over spheres, built on the device.
//
// Replaces Renderer::BuildAccelerationStructures (Core/Renderer.h:160-255):
//   1. centroid bounds (order-preserving integer atomics: exact min/max),
//   2. 30-bit Morton codes of the centroids quantised to 10 bits per axis,
//   3. stable LSD radix sort of (code, original index), 4 passes of 8 bits,
//      one warp per tile, stable ranking with __match_any_sync (small scenes:
//      one block for 1 to 3, a bitonic sort),
//   4. Karras 2012 hierarchy ("Maximizing Parallelism in the Construction of
//      BVHs, Octrees, and k-d Trees"), ties on equal codes broken by index,
//   5. bottom-up refit with per-node arrival counters and treelet
//      restructuring in one pass; leaf boxes are the sphere AABBs rounded
//      outward (__fsub_rd / __fadd_ru, |radius|),
//   6. gather of spheres and materials into Morton (slot) order.
// Every step is integer work or exact float min/max, so the result is
// bit-identical to a host build of the same algorithm.
#include "venu_device.cuh"
#include "venu_internal.h"

#include <algorithm>
#include <chrono>
#include <cstddef>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

namespace venu {
namespace {

constexpr int kMaxTileKeys = 512;  // keys per warp tile, at most (see sort_rounds)
constexpr int kWarpsPerBlock = 8;
constexpr int kRadixBits = 8;
constexpr int kBuckets = 1 << kRadixBits;

__device__ __forceinline__ uint32_t f2u(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float u2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// The hoisted leaves, slots ascending.
struct HoistList {
    uint32_t n;
    int32_t slot[kMaxHoisted];
};

// Build-time control block: centroid bounds (order-preserving encoded),
// the bounds used for quantisation, and the hoisted-sphere list.
struct LbvhCtl {
    uint32_t b0[6];       // all centroids: lo.xyz, hi.xyz
    float bounds[6];      // the same bounds as floats
    uint32_t hoist_cnt;   // huge spheres found
    HoistList hoisted;    // n <= kMaxHoisted, 0 if more than kHoistCandidates
    uint32_t hoist_buf[64];
    uint32_t bad_words;   // child words k_trav_layout had to replace (never, for a sound build)
};
constexpr uint32_t kHoistCandidates = 64;

// A sphere is huge when its radius exceeds a quarter of the largest extent of
// all centroids (the r = 1000 ground sphere of the RTIOW scene).
__device__ __forceinline__ float huge_threshold(const uint32_t* b0) {
    float m = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) m = fmaxf(m, u2f(b0[3 + a]) - u2f(b0[a]));
    return 0.25f * m;
}

// What must start from a known value: the control block, the arrival counters
// and the parent links.  One launch instead of four.
__global__ void k_lbvh_init(LbvhCtl* c, uint32_t n, uint32_t nint, uint32_t* __restrict__ totals,
                            uint32_t* __restrict__ arrive, int32_t* __restrict__ pint, int32_t* __restrict__ pleaf,
                            uint32_t* __restrict__ trace_err) {
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    if (i0 == 0) {
        for (int a = 0; a < 3; ++a) {
            c->b0[a] = 0xffffffffu;
            c->b0[3 + a] = 0u;
        }
        c->hoist_cnt = 0;
        c->hoisted.n = 0;
        c->bad_words = 0;
    }
    if (totals)
        for (uint32_t i = i0; i < 4u * kBuckets; i += step) totals[i] = 0u;
    if (trace_err)
        for (uint32_t i = i0; i < kTraceWords; i += step) trace_err[i] = 0u;
    for (uint32_t i = i0; i < nint; i += step) {
        arrive[i] = 0u;
        pint[i] = -1;
    }
    for (uint32_t i = i0; i < n; i += step) pleaf[i] = -1;
}

// Centroid bounds (exact min/max through order-preserving integer atomics,
// one set a block: a set a warp kept 300k spheres' launch at 40 us).
__global__ void __launch_bounds__(256) k_bounds(const venu_sphere* __restrict__ s, uint32_t n,
                                                uint32_t* __restrict__ bu) {
    __shared__ uint32_t ends[6];
    if (threadIdx.x < 6) ends[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
    __syncthreads();
    uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0, 0, 0};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            uint32_t u = f2u(s[i].center[a]);
            lo[a] = min(lo[a], u);
            hi[a] = max(hi[a], u);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&ends[a], l);
            atomicMax(&ends[3 + a], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(bu + threadIdx.x, ends[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(bu + threadIdx.x, ends[threadIdx.x]);
}

// Karras's bit spreading: bit i of v goes to bit 3i.
__device__ __forceinline__ uint32_t spread10(uint32_t v) {
    v &= 0x3ffu;
    v = (v * 0x00010001u) & 0xFF0000FFu;
    v = (v * 0x00000101u) & 0x0F00F00Fu;
    v = (v * 0x00000011u) & 0xC30C30C3u;
    v = (v * 0x00000005u) & 0x49249249u;
    return v;
}
__device__ __forceinline__ uint32_t quant10(float c, float lo, float ext) {
    if (!(ext > 0.0f)) return 0;
    float t = (c - lo) / ext;
    float f = t * 1024.0f;
    f = fminf(fmaxf(f, 0.0f), 1023.0f);
    return (uint32_t)f;
}

// Morton codes quantised to the centroid bounds with one scale for all three
// axes (the largest extent), so cells stay cubic: a flat scene is split flat
// instead of its thin axis being stretched over 1024 levels.  (Measured on
// the oracle: 27 % fewer box tests per segment on a 200 000-sphere scene and
// 18 % on 1 M spheres than per-axis scaling, equal on the RTIOW scene.)
// Also counts the digits of each radix pass (the same for all orders).
__global__ void __launch_bounds__(256) k_morton(const venu_sphere* __restrict__ s, uint32_t n, LbvhCtl* c,
                                                uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                uint32_t* __restrict__ totals) {
    __shared__ uint32_t digits[4 * kBuckets];
    for (int i = threadIdx.x; i < 4 * kBuckets; i += blockDim.x) digits[i] = 0u;
    __syncthreads();
    const uint32_t* bu = c->b0;
    float lo[3], ext = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        lo[a] = u2f(bu[a]);
        float hi = u2f(bu[3 + a]);
        ext = fmaxf(ext, hi - lo[a]);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            c->bounds[a] = lo[a];
            c->bounds[3 + a] = hi;
        }
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t qx = quant10(s[i].center[0], lo[0], ext);
        uint32_t qy = quant10(s[i].center[1], lo[1], ext);
        uint32_t qz = quant10(s[i].center[2], lo[2], ext);
        const uint32_t key = (spread10(qx) << 2) | (spread10(qy) << 1) | spread10(qz);
        keys[i] = key;
        vals[i] = i;
#pragma unroll
        for (int d = 0; d < 4; ++d) atomicAdd(&digits[d * kBuckets + ((key >> (8 * d)) & (kBuckets - 1))], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * kBuckets; i += blockDim.x)
        if (digits[i]) atomicAdd(totals + i, digits[i]);
}

// Bounds, codes and sort of a small scene in one block (in place of 15
// launches, each of which costs more than its work here): a bitonic sort of
// (code, index) pairs in shared memory, whose order is that of the stable
// sort by code.  Builds of 485 / 2000 / 4000 spheres with it 134 / 178 / 207 us;
// 485 and 2000 through the general path 204 / 254.
constexpr uint32_t kSmallScene = 4096;
__global__ void __launch_bounds__(1024) k_small_codes(const venu_sphere* __restrict__ s, uint32_t n, uint32_t n2,
                                                      LbvhCtl* c, uint32_t* __restrict__ keys,
                                                      uint32_t* __restrict__ vals) {
    __shared__ unsigned long long pair[kSmallScene];
    __shared__ uint32_t ends[6];
    const uint32_t t = threadIdx.x, nt = blockDim.x;
    if (t < 6) ends[t] = t < 3 ? 0xffffffffu : 0u;
    __syncthreads();
    uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0, 0, 0};
    for (uint32_t i = t; i < n; i += nt)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const uint32_t u = f2u(s[i].center[a]);
            lo[a] = min(lo[a], u);
            hi[a] = max(hi[a], u);
        }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
        if ((t & 31u) == 0) {
            atomicMin(&ends[a], l);
            atomicMax(&ends[3 + a], h);
        }
    }
    __syncthreads();
    float base[3], ext = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        base[a] = u2f(ends[a]);
        ext = fmaxf(ext, u2f(ends[3 + a]) - base[a]);
    }
    if (t < 6) {
        c->b0[t] = ends[t];
        c->bounds[t] = u2f(ends[t]);
    }
    for (uint32_t i = t; i < n2; i += nt) {
        unsigned long long v = ~0ull;
        if (i < n) {
            const uint32_t qx = quant10(s[i].center[0], base[0], ext);
            const uint32_t qy = quant10(s[i].center[1], base[1], ext);
            const uint32_t qz = quant10(s[i].center[2], base[2], ext);
            v = (unsigned long long)((spread10(qx) << 2) | (spread10(qy) << 1) | spread10(qz)) << 32 | i;
        }
        pair[i] = v;
    }
    for (uint32_t k = 2; k <= n2; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            __syncthreads();
            for (uint32_t q = t; q < n2 / 2; q += nt) {
                const uint32_t i = (q & ~(j - 1u)) << 1 | (q & (j - 1u));
                const unsigned long long x = pair[i], y = pair[i + j];
                if ((x > y) == ((i & k) == 0u)) {
                    pair[i] = y;
                    pair[i + j] = x;
                }
            }
        }
    __syncthreads();
    for (uint32_t i = t; i < n; i += nt) {
        keys[i] = (uint32_t)(pair[i] >> 32);
        vals[i] = (uint32_t)pair[i];
    }
}

// The (at most 4) lowest huge slots are hoisted and their leaf words flagged;
// with more than 64 huge spheres nothing is hoisted (deterministically).
__global__ void k_hoist_finalize(LbvhCtl* c, const int32_t* __restrict__ pleaf, float4* nodes, uint32_t n) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t cnt = c->hoist_cnt;
    if (cnt == 0 || cnt > kHoistCandidates) {
        c->hoisted.n = 0;
        return;
    }
    uint32_t buf[kHoistCandidates];
    for (uint32_t i = 0; i < cnt; ++i) buf[i] = c->hoist_buf[i];
    for (uint32_t i = 1; i < cnt; ++i) {  // insertion sort
        uint32_t v = buf[i], j = i;
        while (j > 0 && buf[j - 1] > v) {
            buf[j] = buf[j - 1];
            --j;
        }
        buf[j] = v;
    }
    const uint32_t nh = cnt < (uint32_t)kMaxHoisted ? cnt : (uint32_t)kMaxHoisted;
    for (uint32_t i = 0; i < nh; ++i) {
        const uint32_t k = buf[i];
        const int32_t p = pleaf[k];
        c->hoisted.slot[i] = (int32_t)k;
        if (p < 0 || (uint32_t)p >= n - 1) continue;
        const int32_t want = (int32_t)k | kLeaf;
        if (__float_as_int(nodes[2 * p].w) == want)
            nodes[2 * p].w = __int_as_float(want | kHoisted);
        else if (__float_as_int(nodes[2 * p + 1].w) == want)
            nodes[2 * p + 1].w = __int_as_float(want | kHoisted);
    }
    c->hoisted.n = nh;
}

// Per-tile digit histogram, digit-major: hist[d * ntiles + tile].
__global__ void k_hist(const uint32_t* __restrict__ keys, uint32_t n, int shift, uint32_t ntiles, uint32_t rounds,
                       uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[kWarpsPerBlock][kBuckets];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x * kWarpsPerBlock + w;
    for (int d = lane; d < kBuckets; d += 32) cnt[w][d] = 0;
    __syncwarp();
    if (tile < ntiles) {
        for (uint32_t j = 0; j < rounds; ++j) {
            uint32_t idx = (tile * rounds + j) * 32 + lane;
            if (idx < n) atomicAdd(&cnt[w][(keys[idx] >> shift) & (kBuckets - 1)], 1u);
        }
        __syncwarp();
        for (int d = lane; d < kBuckets; d += 32) hist[(size_t)d * ntiles + tile] = cnt[w][d];
    }
}

// Exclusive scan of `total` counters in place (one block of 1024 threads).
__global__ void k_scan(uint32_t* __restrict__ a, uint32_t total) {
    __shared__ uint32_t part[1024];
    const uint32_t t = threadIdx.x;
    const uint32_t per = (total + blockDim.x - 1) / blockDim.x;
    const uint32_t b = t * per, e = min(total, b + per);
    uint32_t sum = 0;
    for (uint32_t i = b; i < e; ++i) sum += a[i];
    part[t] = sum;
    __syncthreads();
    for (uint32_t off = 1; off < blockDim.x; off <<= 1) {
        uint32_t v = t >= off ? part[t - off] : 0;
        __syncthreads();
        part[t] += v;
        __syncthreads();
    }
    uint32_t run = part[t] - sum;  // exclusive prefix of this thread's chunk
    for (uint32_t i = b; i < e; ++i) {
        uint32_t v = a[i];
        a[i] = run;
        run += v;
    }
}

// The radix pass's offsets: block d turns row d of the tile histogram into
// where each tile's keys of digit d go, from the digit totals and a scan of
// its row.  (One block scanning all 256 x ntiles counters took 17 us of a 40k
// build and 129 us of a 300k one, per pass.)
__global__ void __launch_bounds__(256) k_scan_rows(uint32_t* __restrict__ hist, uint32_t ntiles,
                                                   const uint32_t* __restrict__ totals) {
    __shared__ uint32_t part[8], below[8];
    const uint32_t t = threadIdx.x, lane = t & 31u, w = t >> 5, d = blockIdx.x;
    uint32_t* const row = hist + (size_t)d * ntiles;
    const uint32_t per = (ntiles + 255u) / 256u;
    const uint32_t b = min(ntiles, t * per), e = min(ntiles, b + per);
    uint32_t sum = 0;
    for (uint32_t i = b; i < e; ++i) sum += row[i];
    uint32_t incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= (uint32_t)off) incl += v;
    }
    const uint32_t under = __reduce_add_sync(0xffffffffu, t < d ? totals[t] : 0u);
    if (lane == 31) part[w] = incl;
    if (lane == 0) below[w] = under;
    __syncthreads();
    uint32_t run = incl - sum;
#pragma unroll
    for (uint32_t v = 0; v < 8; ++v) {
        run += below[v];
        if (v < w) run += part[v];
    }
    for (uint32_t i = b; i < e; ++i) {
        const uint32_t v = row[i];
        row[i] = run;
        run += v;
    }
}

// Stable scatter: keys of a tile are ranked in tile order within their digit.
__global__ void k_scatter(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint32_t n,
                          int shift, uint32_t ntiles, uint32_t rounds, const uint32_t* __restrict__ offs,
                          uint32_t* __restrict__ kout, uint32_t* __restrict__ vout) {
    __shared__ uint32_t base[kWarpsPerBlock][kBuckets];
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t tile = blockIdx.x * kWarpsPerBlock + w;
    if (tile >= ntiles) return;  // whole warp leaves together
    for (int d = lane; d < kBuckets; d += 32) base[w][d] = offs[(size_t)d * ntiles + tile];
    __syncwarp();
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t j = 0; j < rounds; ++j) {
        uint32_t idx = (tile * rounds + j) * 32 + lane;
        bool valid = idx < n;
        uint32_t k = valid ? kin[idx] : 0u;
        uint32_t d = valid ? ((k >> shift) & (kBuckets - 1)) : (uint32_t)kBuckets + lane;
        uint32_t peers = __match_any_sync(0xffffffffu, d);
        uint32_t rank = __popc(peers & lt);
        uint32_t pos = valid ? base[w][d] + rank : 0u;
        __syncwarp();
        if (valid && rank == 0) base[w][d] += __popc(peers);
        __syncwarp();
        if (valid) {
            kout[pos] = k;
            vout[pos] = vin[idx];
        }
    }
}

__device__ __forceinline__ int delta(const uint32_t* __restrict__ k, int n, int i, int j) {
    if (j < 0 || j > n - 1) return -1;
    uint32_t a = k[i], b = k[j];
    if (a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}

// One thread per internal node i in [0, n-2].
__global__ void k_karras(const uint32_t* __restrict__ keys, int n, float4* __restrict__ nodes,
                         int32_t* __restrict__ parent_int, int32_t* __restrict__ parent_leaf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(keys, n, i, i + 1) - delta(keys, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(keys, n, i, i - d);
    int lmax = 2;
    while (delta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
    int l = 0;
    for (int t = lmax / 2; t >= 1; t /= 2)
        if (delta(keys, n, i, i + (l + t) * d) > dmin) l += t;
    int j = i + l * d;
    int dnode = delta(keys, n, i, j);
    int s = 0;
    int t = l;
    do {
        t = (t + 1) >> 1;  // ceil(l/2), ceil(l/4), ..., 1
        if (delta(keys, n, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int gamma = i + s * d + min(d, 0);
    int left = (min(i, j) == gamma) ? (gamma | kLeaf) : gamma;
    int right = (max(i, j) == gamma + 1) ? ((gamma + 1) | kLeaf) : gamma + 1;
    nodes[2 * i].w = __int_as_float(left);
    nodes[2 * i + 1].w = __int_as_float(right);
    if (left & kLeaf) parent_leaf[left & ~kLeaf] = i; else parent_int[left] = i;
    if (right & kLeaf) parent_leaf[right & ~kLeaf] = i; else parent_int[right] = i;
    if (i == 0) parent_int[0] = -1;
}

// Arrival at a node: publishes what this thread (and, before a __syncwarp,
// its warp) has written, and sees what the earlier arrival published.
__device__ __forceinline__ uint32_t arrive_acq_rel(uint32_t* counter) {
    uint32_t old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}

// Box of a leaf: the sphere's AABB with |radius|, rounded outwards.  An
// exactly-zero difference rounds down to -0.0; "+ 0.0f" makes it +0.0 (still a
// lower bound) so boxes never carry a signed zero.
__device__ __forceinline__ void leaf_box(float4 s4, float4& lo, float4& hi) {
    const float r = fabsf(s4.w);
    lo = make_float4(__fsub_rd(s4.x, r) + 0.0f, __fsub_rd(s4.y, r) + 0.0f, __fsub_rd(s4.z, r) + 0.0f, 0.0f);
    hi = make_float4(__fadd_ru(s4.x, r), __fadd_ru(s4.y, r), __fadd_ru(s4.z, r), 0.0f);
}

// Bottom-up refit of moved spheres (sph: slot order).  The second thread to
// arrive at a node (counters from 0, see k_gather) computes its box; the
// arrivals publish the children's boxes, which are read back through L2
// (__ldcg).  The tree itself does not change, so a node's child
// words and parent are read beside its arrival.  Leaf words may carry the
// hoisted flag.
__global__ void k_refit(const float4* __restrict__ sph, int n, float4* nodes, const int32_t* __restrict__ parent_int,
                        const int32_t* __restrict__ parent_leaf, uint32_t* __restrict__ arrive) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int p = parent_leaf[k];
    // A Karras tree over unique (code, index) keys is at most 63 levels deep;
    // the bound only guards against a corrupt parent chain.
    for (int level = 0; p >= 0 && p < n - 1 && level < 128; ++level) {
        const int32_t cl = __float_as_int(__ldcg(&nodes[2 * p].w));
        const int32_t cr = __float_as_int(__ldcg(&nodes[2 * p + 1].w));
        const int32_t up = parent_int[p];
        if (arrive_acq_rel(arrive + p) == 0u) return;
        const bool ok_l = (cl & kLeaf) ? (cl & kSlotMask) < n : cl < n - 1;
        const bool ok_r = (cr & kLeaf) ? (cr & kSlotMask) < n : cr < n - 1;
        if (!ok_l || !ok_r) return;
        float4 l0, h0, l1, h1;
        if (cl & kLeaf) {
            leaf_box(sph[cl & kSlotMask], l0, h0);
        } else {
            l0 = __ldcg(nodes + 2 * cl);
            h0 = __ldcg(nodes + 2 * cl + 1);
        }
        if (cr & kLeaf) {
            leaf_box(sph[cr & kSlotMask], l1, h1);
        } else {
            l1 = __ldcg(nodes + 2 * cr);
            h1 = __ldcg(nodes + 2 * cr + 1);
        }
        nodes[2 * p] = make_float4(fminf(l0.x, l1.x), fminf(l0.y, l1.y), fminf(l0.z, l1.z), __int_as_float(cl));
        nodes[2 * p + 1] = make_float4(fmaxf(h0.x, h1.x), fmaxf(h0.y, h1.y), fmaxf(h0.z, h1.z), __int_as_float(cr));
        p = up;
    }
}

// ---------------------------------------------------------------------------
// Refit and treelet restructuring (Karras & Aila, HPG 2013) in one bottom-up
// pass: at every internal node N, once both of its subtrees are final, its
// box is made and a treelet of up to 7 leaves is grown from N's children by
// opening the internal treelet leaf with the largest surface area (first on
// ties); a dynamic program over the 2^7 subsets finds the topology with the
// least total internal surface area, and the treelet is rewired that way if
// that is strictly less than its current total.  Leaves keep their Morton
// slots, N stays the treelet root, the treelet's internal nodes are reused in
// the order they were opened and handed out in depth-first order of the new
// topology.  Same arithmetic, same order as the host LBVH of the oracle, so
// the tree stays bit-exact.
//
// Small scenes are bound by the chain of dependent steps from a leaf to the
// root, large ones by issue; both by the work of one treelet.  So a node's
// record is read once (its box and its child words are the same 32 bytes),
// the growth step is one load and one warp maximum, the 966 (subset,
// partition) pairs of the program are spread over the lanes by subset size
// (about 45 evaluations deep instead of 180), the rewired nodes are written
// by a lane each, and a node whose children are both leaves needs no warp.
// Whole builds against the earlier form (one lane a subset, a refit pass
// before): 485 spheres 530 -> 204 us, 40k 904 -> 420, 300k 2229 -> 1228,
// 1M 5725 -> 3285.
// ---------------------------------------------------------------------------
constexpr int kTreeletLeaves = 7;

// The subsets of 7 entries with 2 .. 7 members, by size.
struct SubsetTable {
    uint8_t s[120];
};
constexpr SubsetTable make_subsets() {
    SubsetTable t{};
    int at = 0;
    for (int k = 2; k <= kTreeletLeaves; ++k)
        for (int S = 1; S < (1 << kTreeletLeaves); ++S) {
            int c = 0;
            for (int b = 0; b < kTreeletLeaves; ++b) c += S >> b & 1;
            if (c == k) t.s[at++] = (uint8_t)S;
        }
    return t;
}
__device__ const SubsetTable kSubsets = make_subsets();
// sizes 2, 3, 4, 5, 6, 7: 21, 35, 35, 21, 7, 1 subsets
constexpr int kSub2 = 0, kSub3 = 21, kSub4 = 56, kSub5 = 91, kSub6 = 112;

struct TBox {
    float lo[3], hi[3];
};

__device__ __forceinline__ float tbox_area(const TBox& b) {
    const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return 2.0f * ((dx * dy + dy * dz) + dz * dx);
}

__device__ __forceinline__ void tbox_add(TBox& u, const TBox& b) {
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        u.lo[ax] = fminf(u.lo[ax], b.lo[ax]);
        u.hi[ax] = fmaxf(u.hi[ax], b.hi[ax]);
    }
}

// An entry of a treelet: a child word, its box, and its own child words when
// it is an internal node.
struct TEntry {
    TBox b;
    int32_t word, left, right;
};

__device__ __forceinline__ void tentry_load(TEntry& e, const float4* nodes, const float4* __restrict__ sph,
                                            int32_t word) {
    float4 lo, hi;
    if (word & kLeaf) {
        leaf_box(sph[word & kSlotMask], lo, hi);
    } else {
        lo = __ldcg(nodes + 2 * (size_t)word);
        hi = __ldcg(nodes + 2 * (size_t)word + 1);
    }
    e.word = word;
    e.b.lo[0] = lo.x;
    e.b.lo[1] = lo.y;
    e.b.lo[2] = lo.z;
    e.b.hi[0] = hi.x;
    e.b.hi[1] = hi.y;
    e.b.hi[2] = hi.z;
    e.left = __float_as_int(lo.w);
    e.right = __float_as_int(hi.w);
}

__device__ __forceinline__ bool word_ok(int32_t w, int n) {
    return (w & kLeaf) ? (w & kSlotMask) < n : (uint32_t)w < (uint32_t)(n - 1);
}

// A warp's shared memory.
struct TreeletSmem {
    float4 box[kTreeletLeaves][2];
    float area[1 << kTreeletLeaves];
    float cost[1 << kTreeletLeaves];
    uint8_t split[1 << kTreeletLeaves];
};

// One partition of S: cost of its two sides; kept when strictly less.
__device__ __forceinline__ void try_partition(const TreeletSmem& T, int S, int P, float& bc, int& bp) {
    const float c = T.cost[P] + T.cost[S ^ P];
    if (c < bc) {
        bc = c;
        bp = P;
    }
}

// The least partition of S by one lane: the side with the lowest member runs
// over low | Q, Q the proper subsets of the rest, largest first.
__device__ __forceinline__ void solve_subset(TreeletSmem& T, int S) {
    const int low = S & -S, rest = S ^ low;
    float bc = INFINITY;
    int bp = 0;
    for (int Q = (rest - 1) & rest;; Q = (Q - 1) & rest) {
        try_partition(T, S, Q | low, bc, bp);
        if (Q == 0) break;
    }
    T.cost[S] = T.area[S] + bc;
    T.split[S] = (uint8_t)bp;
}

// Restructures the treelet rooted at N with the whole warp.  Lane `who` holds
// N's two children in c0 and c1 and N's area.  Every lane calls it with the
// same N.
__device__ void restructure_treelet_warp(int32_t N, int n, int who, const TEntry& c0, const TEntry& c1, float area_n,
                                         float4* nodes, int32_t* parent_int, int32_t* parent_leaf,
                                         const float4* __restrict__ sph, TreeletSmem& T) {
    constexpr uint32_t kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    // lane i < nl holds entry i, lane i < ni internal node i of the treelet
    TEntry e;
    {
        const bool second = lane == 1;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const float l0 = __shfl_sync(kAll, c0.b.lo[ax], who), l1 = __shfl_sync(kAll, c1.b.lo[ax], who);
            const float h0 = __shfl_sync(kAll, c0.b.hi[ax], who), h1 = __shfl_sync(kAll, c1.b.hi[ax], who);
            e.b.lo[ax] = second ? l1 : l0;
            e.b.hi[ax] = second ? h1 : h0;
        }
        const int32_t w0 = __shfl_sync(kAll, c0.word, who), w1 = __shfl_sync(kAll, c1.word, who);
        const int32_t a0 = __shfl_sync(kAll, c0.left, who), a1 = __shfl_sync(kAll, c1.left, who);
        const int32_t b0 = __shfl_sync(kAll, c0.right, who), b1 = __shfl_sync(kAll, c1.right, who);
        e.word = second ? w1 : w0;
        e.left = second ? a1 : a0;
        e.right = second ? b1 : b0;
    }
    float current = 0.0f + __shfl_sync(kAll, area_n, who);  // the treelet's internal area, in the order opened
    int32_t my_int = N;
    int nl = 2, ni = 1;
    float area = lane < 2 && !(e.word & kLeaf) ? tbox_area(e.b) : -1.0f;
    while (nl < kTreeletLeaves) {
        const uint32_t key = area >= 0.0f ? __float_as_uint(area) + 1u : 0u;  // orders like the area
        const uint32_t top = __reduce_max_sync(kAll, key);
        if (top == 0u) break;  // no internal entry left
        const int bi = __ffs(__ballot_sync(kAll, key == top)) - 1;
        current = current + __uint_as_float(top - 1u);
        const int32_t c = __shfl_sync(kAll, e.word, bi);
        const int32_t left = __shfl_sync(kAll, e.left, bi), right = __shfl_sync(kAll, e.right, bi);
        if (!word_ok(left, n) || !word_ok(right, n)) return;  // never for a sound tree
        if (lane == ni) my_int = c;
        ++ni;
        if (lane == bi || lane == nl) {
            tentry_load(e, nodes, sph, lane == bi ? left : right);
            area = (e.word & kLeaf) ? -1.0f : tbox_area(e.b);
        }
        ++nl;
    }
    if (nl < 3) return;  // the same decision in every lane
    const int full = (1 << nl) - 1;
    __syncwarp();  // the previous treelet's reads of T are done
    if (lane < nl) {
        T.box[lane][0] = make_float4(e.b.lo[0], e.b.lo[1], e.b.lo[2], 0.0f);
        T.box[lane][1] = make_float4(e.b.hi[0], e.b.hi[1], e.b.hi[2], 0.0f);
        T.cost[1 << lane] = 0.0f;
    }
    __syncwarp();
    auto box_of = [&](int i) {
        const float4 lo = T.box[i][0], hi = T.box[i][1];
        return TBox{{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
    };
    // areas of the subsets: the members among the first five from the lane's
    // bits, then the four choices of the last two
    {
        TBox u{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
#pragma unroll
        for (int i = 0; i < 5; ++i)
            if (i < nl && (lane >> i & 1)) tbox_add(u, box_of(i));
        if (lane <= full && lane) T.area[lane] = tbox_area(u);
        if (nl > 5) {
            TBox v = u;
            tbox_add(v, box_of(5));
            T.area[32 | lane] = tbox_area(v);
            if (nl > 6) {
                tbox_add(u, box_of(6));
                T.area[64 | lane] = tbox_area(u);
                tbox_add(v, box_of(6));
                T.area[96 | lane] = tbox_area(v);
            }
        }
    }
    __syncwarp();
    // subsets by size; those with entries the treelet does not have are skipped
    if (lane < 21) {
        const int S = kSubsets.s[kSub2 + lane];
        if (S <= full) {
            T.cost[S] = T.area[S] + 0.0f;
            T.split[S] = (uint8_t)(S & -S);
        }
    }
    __syncwarp();
    for (int i = lane; i < 35; i += 32) {
        const int S = kSubsets.s[kSub3 + i];
        if (S <= full) solve_subset(T, S);
    }
    __syncwarp();
    if (nl >= 4) {
        for (int i = lane; i < 35; i += 32) {
            const int S = kSubsets.s[kSub4 + i];
            if (S <= full) solve_subset(T, S);
        }
        __syncwarp();
    }
    if (nl >= 5) {
        if (lane < 21) {
            const int S = kSubsets.s[kSub5 + lane];
            if (S <= full) solve_subset(T, S);
        }
        __syncwarp();
    }
    if (nl >= 6) {  // 7 subsets of 31 partitions: four lanes each
        const int S = kSubsets.s[kSub6 + min(lane >> 2, 6)];
        const int low = S & -S, rest = S ^ low;
        float bc = INFINITY;
        int bp = 0;
        if (S <= full && lane < 28) {
            int Q = rest;
            for (int j = lane & 3; j >= 0; --j) Q = (Q - 1) & rest;
            for (int i = lane & 3; i < 31; i += 4) {
                try_partition(T, S, Q | low, bc, bp);
#pragma unroll
                for (int j = 0; j < 4; ++j) Q = (Q - 1) & rest;
            }
        }
#pragma unroll
        for (int off = 1; off <= 2; off <<= 1) {
            const float oc = __shfl_xor_sync(kAll, bc, off);
            const int op = __shfl_xor_sync(kAll, bp, off);
            if (oc < bc || (oc == bc && op > bp)) {  // the first of equal ones: the largest side
                bc = oc;
                bp = op;
            }
        }
        if (S <= full && lane < 28 && (lane & 3) == 0) {
            T.cost[S] = T.area[S] + bc;
            T.split[S] = (uint8_t)bp;
        }
        __syncwarp();
    }
    if (nl == 7) {  // 63 partitions of the whole set over the warp
        float bc = INFINITY;
        int bp = 0;
        try_partition(T, full, ((62 - lane) << 1) | 1, bc, bp);
        if (lane < 31) try_partition(T, full, ((30 - lane) << 1) | 1, bc, bp);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float oc = __shfl_xor_sync(kAll, bc, off);
            const int op = __shfl_xor_sync(kAll, bp, off);
            if (oc < bc || (oc == bc && op > bp)) {
                bc = oc;
                bp = op;
            }
        }
        if (lane == 0) {
            T.cost[full] = T.area[full] + bc;
            T.split[full] = (uint8_t)bp;
        }
        __syncwarp();
    }
    if (!(T.cost[full] < current)) return;
    // order: byte i is the subset of the i-th internal node in depth-first
    // preorder; it is given internal node i
    unsigned long long order = 0, stack = (unsigned long long)full;
    int no = 0;
    while (stack) {
        const int S = (int)(stack & 0xffu);
        stack >>= 8;
        order |= (unsigned long long)S << (8 * no++);
        const int P = T.split[S], O = S ^ P;
        if (O & (O - 1)) stack = stack << 8 | (unsigned)O;
        if (P & (P - 1)) stack = stack << 8 | (unsigned)P;
    }
    const int S = lane < no ? (int)(order >> (8 * lane) & 0xffu) : full;
    const int P = T.split[S], O = S ^ P;
    auto word = [&](int X) -> int32_t {
        int at = 0;  // the internal node that X is given
        for (int i = 1; i < no; ++i)
            if ((int)(order >> (8 * i) & 0xffu) == X) at = i;
        const int32_t leaf_word = __shfl_sync(kAll, e.word, __ffs(X) - 1);
        const int32_t int_word = __shfl_sync(kAll, my_int, at);
        return (X & (X - 1)) == 0 ? leaf_word : int_word;
    };
    const int32_t l = word(P), r = word(O);
    TBox u{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
    for (int i = 0; i < nl; ++i)
        if (S >> i & 1) tbox_add(u, box_of(i));
    if (lane < no) {
        const int32_t me = my_int;
        nodes[2 * (size_t)me] = make_float4(u.lo[0], u.lo[1], u.lo[2], __int_as_float(l));
        nodes[2 * (size_t)me + 1] = make_float4(u.hi[0], u.hi[1], u.hi[2], __int_as_float(r));
        if (l & kLeaf) parent_leaf[l & kSlotMask] = me;
        else parent_int[l] = me;
        if (r & kLeaf) parent_leaf[r & kSlotMask] = me;
        else parent_int[r] = me;
    }
}

// A warp starts from `per_warp` leaves (a power of two, at most 32), one a
// lane; each walks up as in k_refit, and the lane that reaches a node second
// makes its box from its final children.  Nodes that need restructuring are
// then served one after another by the whole warp: the lanes stay in the
// loop until none of them is walking.  Fewer leaves a warp make fewer nodes
// to serve in turn (31 of them for 32 leaves) and more warps.
constexpr int kTreeletBlock = 128;
__global__ void __launch_bounds__(kTreeletBlock)
    k_treelets(const float4* __restrict__ sph, int n, int per_warp, float4* nodes, int32_t* parent_int,
               int32_t* parent_leaf, uint32_t* __restrict__ arrive) {
    __shared__ TreeletSmem smem[kTreeletBlock / 32];
    TreeletSmem& T = smem[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long long first = (long long)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per_warp;
    bool walking = lane < per_warp && first + lane < n;
    int p = walking ? parent_leaf[(int)first + lane] : -1;
    for (int level = 0; level < 128; ++level) {
        bool want = false;
        int up = -1;
        TEntry c0{}, c1{};
        float area = 0.0f;
        if (walking) {
            if (p < 0 || p >= n - 1) {
                walking = false;
            } else {
                // p's child words and its parent stay what they are until p is
                // restructured, or an ancestor: read beside the arrival
                const int32_t w0 = __float_as_int(__ldcg(&nodes[2 * (size_t)p].w));
                const int32_t w1 = __float_as_int(__ldcg(&nodes[2 * (size_t)p + 1].w));
                up = __ldcg(parent_int + p);
                if (arrive_acq_rel(arrive + p) == 0u) {
                    walking = false;  // the other subtree is not final yet
                } else {
                    if (word_ok(w0, n) && word_ok(w1, n)) {
                        tentry_load(c0, nodes, sph, w0);
                        tentry_load(c1, nodes, sph, w1);
                        TBox u = c0.b;
                        tbox_add(u, c1.b);
                        nodes[2 * (size_t)p] = make_float4(u.lo[0], u.lo[1], u.lo[2], __int_as_float(w0));
                        nodes[2 * (size_t)p + 1] = make_float4(u.hi[0], u.hi[1], u.hi[2], __int_as_float(w1));
                        area = tbox_area(u);
                        want = !(w0 & kLeaf) || !(w1 & kLeaf);
                    } else {
                        walking = false;  // never for a sound tree
                    }
                }
            }
        }
        __syncwarp();
        for (uint32_t m = __ballot_sync(0xffffffffu, want); m; m &= m - 1u) {
            const int who = __ffs(m) - 1;
            const int32_t q = __shfl_sync(0xffffffffu, p, who);
            restructure_treelet_warp(q, n, who, c0, c1, area, nodes, parent_int, parent_leaf, sph, T);
        }
        // the rewiring by the other lanes comes before this lane's releasing
        // arrival at the parent
        __syncwarp();
        p = up;
        if (!__any_sync(0xffffffffu, walking)) break;
    }
}

// Slot-ordered sphere / material / meta records.  ids may alias meta (a
// refit regathers from the meta words): each thread reads its slot's word
// before writing it.  c (builds only): huge spheres become candidates for
// hoisting (unordered, at most 64).  arrive (refits only): the n - 1 arrival
// counters, cleared for the refit that follows.
__global__ void k_gather(const venu_sphere* __restrict__ s, const uint32_t* ids, uint32_t id_mask, uint32_t n,
                         float4* __restrict__ sph, float4* __restrict__ mat, uint32_t* meta, LbvhCtl* c,
                         uint32_t* __restrict__ arrive) {
    uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    if (arrive && k < n - 1u) arrive[k] = 0u;
    uint32_t id = ids[k] & id_mask;
    const venu_sphere& sp = s[id];
    uint32_t type = sp.material > 2u ? 2u : sp.material;
    sph[k] = make_float4(sp.center[0], sp.center[1], sp.center[2], sp.radius);
    float param = type == 1u ? sp.fuzz : (type == 2u ? sp.ir : 0.0f);
    mat[k] = make_float4(sp.albedo[0], sp.albedo[1], sp.albedo[2], param);
    meta[k] = id | (type << 30);
    if (c && fabsf(sp.radius) > huge_threshold(c->b0)) {
        const uint32_t i = atomicAdd(&c->hoist_cnt, 1u);
        if (i < kHoistCandidates) c->hoist_buf[i] = k;
    }
}

// ---------------------------------------------------------------------------
// Traversal layout: internal node p becomes one 64-byte record holding both
// children, child c in the 32 bytes at float4s 4p + 2c and 4p + 2c + 1:
//   {c.x, c.y, h.x, h.y}, {c.z, h.z, word, 0}
// with the centre and the half extents of the child's box (an internal
// node's, or a leaf's sphere box rounded outwards) and its word (leaf and
// hoisted flags kept).  A step of the traversal then reads one record with
// two 32-byte loads instead of two boxes at two addresses, tests nodes and
// leaves by the same instructions, and finds the operands of the packed FMAs
// in adjacent registers.  c +- h encloses the box widened by e (the fast
// walk's bound, venu_device.cuh) under any rounding.  The canonical nodes
// array stays the exported form.
//
// Behind the n - 1 records stands the root's: {c.x, c.y, h.x, h.y},
// {c.z, h.z, 0, 0}, {G, -2^-18 E}.  All boxes are relative to G.
//
// A hoisted leaf is tested before the walk, so its box is empty here
// (h = -inf is never met), and k_hoist_clean takes it out of the boxes above
// it: the r = 1000 ground sphere would otherwise make every box on its way
// to the root one that every ray meets.
//
// Every word written here is in range by construction -- an internal child
// in [1, n-1), a leaf slot below n -- so the traversal needs no per-step
// index checks: a word that is not (which a sound build never produces) is
// replaced by a skipped leaf and counted in *bad.
// ---------------------------------------------------------------------------
// How far the box of a record is widened: 24 2^-24 (Q + E), Q the sum of its
// farthest corner's coordinates (an upper bound of the corner's distance).
__device__ __forceinline__ float widen_of(float3 lo, float3 hi, float E) {
    const float Q = (fmaxf(fabsf(lo.x), fabsf(hi.x)) + fmaxf(fabsf(lo.y), fabsf(hi.y))) + fmaxf(fabsf(lo.z), fabsf(hi.z));
    return (Q + E) * 1.430511474609375e-06f;  // 1.5 2^-20
}

__device__ __forceinline__ void centre_half(float lo, float hi, float e, float& c, float& h) {
    c = 0.5f * lo + 0.5f * hi;
    h = __fadd_ru(fmaxf(__fsub_ru(hi, c), __fsub_ru(c, lo)), e);
    if (!(lo <= hi)) h = __int_as_float(0x7fc00000);  // a NaN box is always met
}

// A box relative to G (rounded outwards), widened, as centres and half extents.
// frame: the third of the root's float4s.
__device__ __forceinline__ void frame_box(float4 lo4, float4 hi4, float4 frame, float3& c, float3& h) {
    const float3 lo = make_float3(__fsub_rd(lo4.x, frame.x), __fsub_rd(lo4.y, frame.y), __fsub_rd(lo4.z, frame.z));
    const float3 hi = make_float3(__fsub_ru(hi4.x, frame.x), __fsub_ru(hi4.y, frame.y), __fsub_ru(hi4.z, frame.z));
    const float e = widen_of(lo, hi, frame.w * -262144.0f);
    centre_half(lo.x, hi.x, e, c.x, h.x);
    centre_half(lo.y, hi.y, e, c.y, h.y);
    centre_half(lo.z, hi.z, e, c.z, h.z);
}

__device__ __forceinline__ void write_child(float4* rec, float4 lo, float4 hi, float4 frame, int32_t w) {
    float3 c, h;
    frame_box(lo, hi, frame, c, h);
    if ((w & kLeaf) && (w & kHoisted)) {
        c = make_float3(0.0f, 0.0f, 0.0f);
        h = make_float3(-INFINITY, -INFINITY, -INFINITY);
    }
    rec[0] = make_float4(c.x, c.y, h.x, h.y);
    rec[1] = make_float4(c.z, h.z, __int_as_float(w), 0.0f);
}

// The value that is left of a warp's samples (two a lane) at the low end, or the
// high one, when `trim` have been taken away there.  At least one is valid.
__device__ float trimmed_end(float a, bool va, float b, bool vb, uint32_t trim, bool high) {
    const uint32_t flip = high ? 0xffffffffu : 0u;
    uint32_t x = va ? f2u(a) ^ flip : 0xffffffffu, y = vb ? f2u(b) ^ flip : 0xffffffffu;
    for (;; --trim) {
        const uint32_t m = __reduce_min_sync(0xffffffffu, min(x, y));
        if (trim == 0u) return u2f(m ^ flip);
        const uint32_t has = __ballot_sync(0xffffffffu, min(x, y) == m);
        if ((threadIdx.x & 31u) == (uint32_t)__ffs(has) - 1u) {
            if (x == m) x = 0xffffffffu;
            else y = 0xffffffffu;
        }
    }
}

// G and E of the records (one warp): 64 spheres evenly spaced in slot order, the
// hoisted and those that are not finite left out.  G is the middle of their
// centres' box and E twice the largest |C - G| + |r|, each once the four outermost
// samples at an end are dropped, so that a few far spheres do not decide.  The
// walk is right with any G and E (venu_device.cuh); they settle how much boxes are
// widened and which rays need a margin.  Twice the radius, because the margin
// takes |p| as the sum of its coordinates, and an origin in a corner of the scene
// should need none: a nearly axis-parallel ray with a margin goes the slow way and
// its warp waits for it (at once the radius: 1M ray queries on 20k spheres 667 ->
// 918 us, 96 uneven jobs 6.88 -> 7.19 ms, 100k moving spheres 2.10 -> 2.23 ms).
__global__ void k_frame(const float4* __restrict__ sph, uint32_t n, const HoistList* __restrict__ ctl_list,
                        HoistList list, float4* __restrict__ frame) {
    const HoistList H = ctl_list ? *ctl_list : list;
    float4 s[2];
    bool ok[2];
    for (int j = 0; j < 2; ++j) {
        const uint32_t k = (uint32_t)((unsigned long long)(2u * threadIdx.x + (uint32_t)j) * n / 64u);
        s[j] = sph[k];
        ok[j] = isfinite(s[j].x) && isfinite(s[j].y) && isfinite(s[j].z) && isfinite(s[j].w);
        for (uint32_t i = 0; i < H.n; ++i) ok[j] = ok[j] && H.slot[i] != (int32_t)k;
    }
    const uint32_t valid = __reduce_add_sync(0xffffffffu, (uint32_t)ok[0] + (uint32_t)ok[1]);
    float4 F = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (valid) {
        const uint32_t trim = min(4u, valid / 4u);
        F.x = 0.5f * trimmed_end(s[0].x, ok[0], s[1].x, ok[1], trim, false) +
              0.5f * trimmed_end(s[0].x, ok[0], s[1].x, ok[1], trim, true);
        F.y = 0.5f * trimmed_end(s[0].y, ok[0], s[1].y, ok[1], trim, false) +
              0.5f * trimmed_end(s[0].y, ok[0], s[1].y, ok[1], trim, true);
        F.z = 0.5f * trimmed_end(s[0].z, ok[0], s[1].z, ok[1], trim, false) +
              0.5f * trimmed_end(s[0].z, ok[0], s[1].z, ok[1], trim, true);
        float q[2];
        for (int j = 0; j < 2; ++j) {
            const float x = s[j].x - F.x, y = s[j].y - F.y, z = s[j].z - F.z;
            q[j] = fminf(sqrtf(x * x + y * y + z * z) + fabsf(s[j].w), 1e30f);
        }
        F.w = -7.62939453125e-06f * trimmed_end(q[0], ok[0], q[1], ok[1], trim, true);  // -2 2^-18
    }
    if (threadIdx.x == 0) *frame = F;
}

__global__ void k_trav_layout(const float4* __restrict__ nodes, const float4* __restrict__ sph, uint32_t n,
                              float4* __restrict__ trav, uint32_t* bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2u * (n - 1u)) return;
    float4* const root = trav + 4 * (size_t)(n - 1u);
    const float4 frame = root[2];
    if (i == 0) {
        float3 c, h;
        frame_box(nodes[0], nodes[1], frame, c, h);
        root[0] = make_float4(c.x, c.y, h.x, h.y);
        root[1] = make_float4(c.z, h.z, 0.0f, 0.0f);
    }
    const uint32_t p = i >> 1, c = i & 1u;
    int32_t w = __float_as_int(nodes[2 * p + c].w);
    const bool ok = (w & kLeaf) ? (uint32_t)(w & kSlotMask) < n && !(w & ~(kLeaf | kHoisted | kSlotMask))
                                : (uint32_t)w - 1u < n - 2u;  // 1 <= w < n-1 (the root is nobody's child)
    if (!ok) {
        w = kLeaf | kHoisted;  // slot 0, never tested
        if (bad) atomicAdd(bad, 1u);
    }
    float4 lo, hi;
    if (w & kLeaf) {
        leaf_box(sph[w & kSlotMask], lo, hi);
    } else {
        lo = nodes[2 * w];
        hi = nodes[2 * w + 1];
    }
    write_child(trav + 4 * (size_t)p + 2 * c, lo, hi, frame, w);
}

// Takes the hoisted leaves out of the boxes of the nodes above them, in the
// records only: one thread per scene walks up from each hoisted leaf; a
// node's box becomes the union of its record's two children (rounded
// outwards), written into its parent's record, or the root's.  Walks of
// several leaves run one after another, so a node above two of them is
// written last by the later walk, with both taken out.  The children's boxes
// are widened for their own coordinates; the union's, which may be larger, take
// 8 2^-24 of their sum more (the slab parameters' 4 2^-24 Q).
__global__ void k_hoist_clean(float4* trav, const int32_t* __restrict__ pint, const int32_t* __restrict__ pleaf,
                              uint32_t n, const HoistList* __restrict__ ctl_list, HoistList list) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const HoistList H = ctl_list ? *ctl_list : list;
    for (uint32_t i = 0; i < H.n; ++i) {
        int32_t p = pleaf[H.slot[i]];
        for (uint32_t level = 0; p >= 0 && (uint32_t)p < n - 1u && level < n; ++level) {
            const float4* T = trav + 4 * (size_t)p;
            const float4 a0 = T[0], b0 = T[1], a1 = T[2], b1 = T[3];
            const int32_t q = pint[p];
            const float c0[3] = {a0.x, a0.y, b0.x}, h0[3] = {a0.z, a0.w, b0.y};
            const float c1[3] = {a1.x, a1.y, b1.x}, h1[3] = {a1.z, a1.w, b1.y};
            float c[3], h[3], far = 0.0f;
            for (int ax = 0; ax < 3; ++ax) {
                if (h0[ax] != -INFINITY && h1[ax] != -INFINITY)
                    far += fmaxf(fabsf(c0[ax]) + h0[ax], fabsf(c1[ax]) + h1[ax]);
            }
            const float e = far * 4.76837158203125e-07f;  // 8 2^-24
            for (int ax = 0; ax < 3; ++ax) {
                const bool e0 = h0[ax] == -INFINITY, e1 = h1[ax] == -INFINITY;
                if (e0) {
                    c[ax] = c1[ax];
                    h[ax] = h1[ax];
                } else if (e1) {
                    c[ax] = c0[ax];
                    h[ax] = h0[ax];
                } else {
                    const float l0 = __fsub_rd(c0[ax], h0[ax]), u0 = __fadd_ru(c0[ax], h0[ax]);
                    const float l1 = __fsub_rd(c1[ax], h1[ax]), u1 = __fadd_ru(c1[ax], h1[ax]);
                    centre_half(fminf(l0, l1), fmaxf(u0, u1), e, c[ax], h[ax]);
                    // a NaN box is always met, and so is every box above it
                    if (!(l0 <= u0) || !(l1 <= u1)) h[ax] = __int_as_float(0x7fc00000);
                }
            }
            if (q >= 0 && (uint32_t)q < n - 1u) {
                float4* Q = trav + 4 * (size_t)q;
                const int side = __float_as_int(Q[1].z) == p ? 0 : (__float_as_int(Q[3].z) == p ? 1 : -1);
                if (side < 0) break;  // never for a sound tree
                Q[2 * side] = make_float4(c[0], c[1], h[0], h[1]);
                reinterpret_cast<float2*>(Q + 2 * side + 1)[0] = make_float2(c[2], h[2]);
            } else {
                float4* root = trav + 4 * (size_t)(n - 1u);
                root[0] = make_float4(c[0], c[1], h[0], h[1]);
                reinterpret_cast<float2*>(root + 1)[0] = make_float2(c[2], h[2]);
            }
            p = q;
        }
    }
}

// The records of a built (or refit) tree, on `st`.  The hoisted slots come
// from the build's control block (ctl_list) or by value.
cudaError_t launch_trav_layout(const float4* nodes, const float4* sph, uint32_t n, float4* trav, const int32_t* pint,
                               const int32_t* pleaf, const HoistList* ctl_list, HoistList list, uint32_t* bad,
                               cudaStream_t st) {
    k_frame<<<1, 32, 0, st>>>(sph, n, ctl_list, list, trav + 4 * (size_t)(n - 1) + 2);
    k_trav_layout<<<(2 * (n - 1) + 255) / 256, 256, 0, st>>>(nodes, sph, n, trav, bad);
    if (ctl_list || list.n) k_hoist_clean<<<1, 32, 0, st>>>(trav, pint, pleaf, n, ctl_list, list);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// The wide traversal tree (renderer variants 4 and 5), collapsed from the
// binary LBVH after its build.  A wide node stands for a binary node r and
// holds up to kWideW (4) of r's descendants: starting from r's two
// children, the internal entry of largest box surface area (the first such
// entry on ties) is replaced by its two children until there are kWideW
// entries or only leaves.  Internal entries become wide nodes themselves.
// The wide nodes are numbered in increasing order of the binary nodes they
// stand for (root first), so the tree is deterministic.  Results do not
// depend on it: the closest hit is the same for any conservative traversal
// (minimum t, ties to the smaller slot).
//
// Node layout (kWideF4 float4s, 128 bytes), structure of arrays over the four
// children:
//   [2a], [2a + 1]  centres and half extents of the child boxes on axis a
//   [6]             child words: an internal child's wide index, or a leaf's
//                   0x80000000 | slot (flags kept)
// The boxes are those of the binary traversal records (widened, hoisted leaves
// taken out); an unused entry's is empty (half extents -inf).
// wide_src[kWideW w + c] is the record of child c, 2 p + side for binary node
// p (or kNoRecord), from which a refit of moved spheres copies the box again.
// ---------------------------------------------------------------------------
constexpr int kWideChildren = kWideW;

__device__ __forceinline__ float box_area(float4 lo, float4 hi) {
    const float dx = hi.x - lo.x, dy = hi.y - lo.y, dz = hi.z - lo.z;
    return dx * dy + dy * dz + dz * dx;
}

constexpr int32_t kNoRecord = -1;

// w: the entries' words, rec: the traversal records they come from.
__device__ int wide_collapse(const float4* __restrict__ nodes, int32_t r, int32_t w[kWideChildren],
                             int32_t rec[kWideChildren]) {
    w[0] = __float_as_int(nodes[2 * r].w);
    w[1] = __float_as_int(nodes[2 * r + 1].w);
    rec[0] = 2 * r;
    rec[1] = 2 * r + 1;
    int cnt = 2;
    while (cnt < kWideChildren) {
        int best = -1;
        float best_a = -1.0f;
        for (int i = 0; i < cnt; ++i) {
            if (w[i] & kLeaf) continue;
            const float a = box_area(nodes[2 * w[i]], nodes[2 * w[i] + 1]);
            if (a > best_a) {
                best_a = a;
                best = i;
            }
        }
        if (best < 0) break;
        const int32_t q = w[best];
        w[best] = __float_as_int(nodes[2 * q].w);
        rec[best] = 2 * q;
        rec[cnt] = 2 * q + 1;
        w[cnt++] = __float_as_int(nodes[2 * q + 1].w);
    }
    return cnt;
}

// One level of the collapse: every binary node of the frontier expands;
// its internal entries are flagged as wide nodes and form the next frontier.
__global__ void k_wide_frontier(const float4* __restrict__ nodes, const int32_t* __restrict__ fin, uint32_t nin,
                                int32_t* __restrict__ fout, uint32_t* __restrict__ nout, uint32_t* __restrict__ flag) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nin) return;
    int32_t w[kWideChildren], rec[kWideChildren];
    const int c = wide_collapse(nodes, fin[i], w, rec);
    for (int j = 0; j < c; ++j) {
        if (w[j] & kLeaf) continue;
        flag[w[j]] = 1u;
        fout[atomicAdd(nout, 1u)] = w[j];
    }
}

// The boxes of a wide node from its children's traversal records.
__device__ void wide_boxes(const float4* __restrict__ trav, const int32_t rec[kWideChildren], float4* __restrict__ W) {
    float c[3][kWideChildren], h[3][kWideChildren];
    for (int j = 0; j < kWideChildren; ++j) {
        float4 a = make_float4(0.0f, 0.0f, -INFINITY, -INFINITY), b = make_float4(0.0f, -INFINITY, 0.0f, 0.0f);
        if (rec[j] != kNoRecord) {
            a = trav[2 * (size_t)rec[j]];
            b = trav[2 * (size_t)rec[j] + 1];
        }
        c[0][j] = a.x; c[1][j] = a.y; c[2][j] = b.x;
        h[0][j] = a.z; h[1][j] = a.w; h[2][j] = b.y;
    }
    for (int a = 0; a < 3; ++a) {
        W[2 * a] = make_float4(c[a][0], c[a][1], c[a][2], c[a][3]);
        W[2 * a + 1] = make_float4(h[a][0], h[a][1], h[a][2], h[a][3]);
    }
}

// One thread per binary internal node; the flagged ones write their wide node.
// idx maps a binary internal node to its wide index.
__global__ void k_wide_write(const float4* __restrict__ nodes, const float4* __restrict__ trav, uint32_t n,
                             const uint32_t* __restrict__ flag, const uint32_t* __restrict__ idx,
                             float4* __restrict__ wide, int32_t* __restrict__ wide_src) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n - 1 || !flag[r]) return;
    int32_t w[kWideChildren], rec[kWideChildren];
    const int c = wide_collapse(nodes, (int32_t)r, w, rec);
    for (int j = 0; j < kWideChildren; ++j) {
        if (j >= c) {
            w[j] = kLeaf | kHoisted;
            rec[j] = kNoRecord;
        } else if (!(w[j] & kLeaf)) {
            w[j] = (int32_t)idx[w[j]];
        }
    }
    const uint32_t k = idx[r];
    for (int j = 0; j < kWideChildren; ++j) wide_src[(size_t)kWideChildren * k + j] = rec[j];
    float4* W = wide + kWideF4 * (size_t)k;
    wide_boxes(trav, rec, W);
    W[6] = make_float4(__int_as_float(w[0]), __int_as_float(w[1]), __int_as_float(w[2]), __int_as_float(w[3]));
    W[7] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Refit of moved spheres: the same topology and words, the boxes from the
// refit traversal records.
__global__ void k_wide_refit(const float4* __restrict__ trav, uint32_t nwide, const int32_t* __restrict__ wide_src,
                             float4* __restrict__ wide) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nwide) return;
    int32_t rec[kWideChildren];
    for (int j = 0; j < kWideChildren; ++j) rec[j] = wide_src[(size_t)kWideChildren * k + j];
    wide_boxes(trav, rec, wide + kWideF4 * (size_t)k);
}

inline uint32_t cdiv(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// Device buffers of one LBVH build: outputs and scratch.  trav may be null
// (the build then stops at the canonical layout).
struct LbvhBuffers {
    float4 *nodes, *trav, *sph, *mat;
    uint32_t *meta, *keys;
    LbvhCtl* ctl;
    uint32_t *keys_alt, *vals, *vals_alt, *hist, *totals, *arrive, *trace_err;
    int32_t *pint, *pleaf;
};

// Bytes of the scratch that only the codes and their sort use (keys_alt,
// vals, vals_alt, hist, totals; each 256-byte aligned).
constexpr size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Keys per lane of a sort tile (a warp's): short tiles while that still
// spreads the keys over the SMs.
uint32_t sort_rounds(uint32_t n) { return n <= 65536u ? 4u : n <= 262144u ? 8u : (uint32_t)kMaxTileKeys / 32u; }

// Leaves a warp of k_treelets starts from: few while that still leaves warps
// to spare (the nodes a warp serves in turn are then the chain that counts),
// 32 once the whole GPU is busy.  Whole builds at 4 / 8 / 16 / 32: 485 spheres
// 204 / 213 / 232 / 250 us, 40k 428 / 420 / 424 / 445, 100k 679 / 646 / 622 /
// 602, 1M 4122 / 3736 / 3459 / 3285.
uint32_t treelet_leaves_per_warp(uint32_t n) {
    uint32_t per = 4;
    while (per < 32u && n / per > 4096u) per *= 2;
    return per;
}

// The whole build, asynchronously on `st`; both venu_scene_create and
// venu_lbvh_build_noalloc run exactly this sequence.
cudaError_t launch_lbvh(const venu_sphere* s, uint32_t n, cudaStream_t st, const LbvhBuffers& B) {
    const uint32_t nint = n > 1 ? n - 1 : 1;
    cudaError_t e = cudaSuccess;
    const uint32_t blocks = std::min(cdiv(n, 256), (uint32_t)(sm_count() * 8));
    k_lbvh_init<<<blocks, 256, 0, st>>>(B.ctl, n, nint, n > kSmallScene ? B.totals : nullptr, B.arrive, B.pint, B.pleaf,
                                        B.trace_err);
    if (n <= kSmallScene) {
        uint32_t n2 = 64;
        while (n2 < n) n2 *= 2;
        k_small_codes<<<1, std::min(n2 / 2, 1024u), 0, st>>>(s, n, n2, B.ctl, B.keys, B.vals);
    } else {
        const uint32_t few = std::min(cdiv(n, 256), (uint32_t)(sm_count() * 2));  // each block ends with atomics
        k_bounds<<<few, 256, 0, st>>>(s, n, B.ctl->b0);
        k_morton<<<few, 256, 0, st>>>(s, n, B.ctl, B.keys, B.vals, B.totals);
        uint32_t *kin = B.keys, *kout = B.keys_alt, *vin = B.vals, *vout = B.vals_alt;
        const uint32_t rounds = sort_rounds(n), ntiles = cdiv(n, 32 * rounds);
        const uint32_t sblocks = cdiv(ntiles, kWarpsPerBlock);
        for (int pass = 0; pass < 4; ++pass) {
            const int shift = pass * kRadixBits;
            k_hist<<<sblocks, 32 * kWarpsPerBlock, 0, st>>>(kin, n, shift, ntiles, rounds, B.hist);
            k_scan_rows<<<kBuckets, 256, 0, st>>>(B.hist, ntiles, B.totals + pass * kBuckets);
            k_scatter<<<sblocks, 32 * kWarpsPerBlock, 0, st>>>(kin, vin, n, shift, ntiles, rounds, B.hist, kout, vout);
            std::swap(kin, kout);
            std::swap(vin, vout);
        }
        // four passes: the sorted codes / ids are back in B.keys / B.vals
    }
    // the gather is the last to read the spheres and the sort's buffers, which
    // may lie where the nodes and the traversal records go
    k_gather<<<cdiv(n, 256), 256, 0, st>>>(s, B.vals, 0xffffffffu, n, B.sph, B.mat, B.meta, n > 1 ? B.ctl : nullptr,
                                         nullptr);
    if (n > 1) {
        k_karras<<<cdiv(n - 1, 256), 256, 0, st>>>(B.keys, (int)n, B.nodes, B.pint, B.pleaf);
        const uint32_t per_warp = treelet_leaves_per_warp(n);
        k_treelets<<<cdiv(cdiv(n, per_warp), kTreeletBlock / 32), kTreeletBlock, 0, st>>>(
            B.sph, (int)n, (int)per_warp, B.nodes, B.pint, B.pleaf, B.arrive);
    }
    if (n > 1) {
        k_hoist_finalize<<<1, 32, 0, st>>>(B.ctl, B.pleaf, B.nodes, n);
        if (B.trav) {
            e = launch_trav_layout(B.nodes, B.sph, n, B.trav, B.pint, B.pleaf, &B.ctl->hoisted, HoistList{},
                                   &B.ctl->bad_words, st);
            if (e != cudaSuccess) return e;
        }
    }
    return cudaGetLastError();
}

}  // namespace

void free_scene(venu_scene* s) {
    if (!s) return;
    cudaFree(s->arena);
    cudaFree(s->wide);
    cudaFree(s->wide_src);
    cudaFree(s->upload);
    if (s->refit_done) cudaEventDestroy(s->refit_done);
    s->refit_done = nullptr;
    s->wide = nullptr;
    s->wide_src = nullptr;
    s->upload = nullptr;
    s->nwide = 0;
    s->arena = nullptr;
    s->parents = nullptr;
    s->arrive = s->trace_err = nullptr;
    s->nodes = s->trav = nullptr;
    s->sph = s->mat = nullptr;
    s->meta = s->keys = nullptr;
}

// The wide tree of a built scene (n > 1): the collapse level by level from
// the root (the host reads each level's size), then one write pass.
venu_status build_wide(const venu_scene* S, cudaStream_t st) {
    const uint32_t n = S->n;
    if (n < 2) return VENU_OK;
    const uint32_t nint = n - 1;
    uint32_t *flag = nullptr, *idx = nullptr, *cnt = nullptr;
    int32_t *fa = nullptr, *fb = nullptr;
    venu_status rc = VENU_OK;
    uint32_t nwide = 0;
#define WSTEP(call)                    \
    do {                               \
        cudaError_t _e = (call);       \
        if (_e != cudaSuccess) {       \
            rc = cuda_fail(_e, #call); \
            goto wdone;                \
        }                              \
    } while (0)
    WSTEP(cudaMalloc(&flag, sizeof(uint32_t) * nint));
    WSTEP(cudaMalloc(&idx, sizeof(uint32_t) * nint));
    WSTEP(cudaMalloc(&cnt, sizeof(uint32_t)));
    WSTEP(cudaMalloc(&fa, sizeof(int32_t) * nint));
    WSTEP(cudaMalloc(&fb, sizeof(int32_t) * nint));
    WSTEP(cudaMemsetAsync(flag, 0, sizeof(uint32_t) * nint, st));
    WSTEP(cudaMemsetAsync(flag, 0x01, 1, st));  // the root
    WSTEP(cudaMemsetAsync(fa, 0, sizeof(int32_t), st));
    {
        // a binary tree over n leaves has fewer than n levels, and each level
        // of the collapse takes at least one of them
        uint32_t nin = 1;
        for (uint32_t level = 0; nin > 0 && level < n; ++level) {
            WSTEP(cudaMemsetAsync(cnt, 0, sizeof(uint32_t), st));
            k_wide_frontier<<<cdiv(nin, 128), 128, 0, st>>>(S->nodes, fa, nin, fb, cnt, flag);
            WSTEP(cudaGetLastError());
            WSTEP(cudaMemcpyAsync(&nin, cnt, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
            WSTEP(cudaStreamSynchronize(st));
            std::swap(fa, fb);
        }
        if (nin > 0) {  // a cyclic (corrupt) binary tree: no wide tree
            set_error("venu_scene_create: the wide-tree collapse did not end");
            rc = VENU_ERR_INVALID;
            goto wdone;
        }
    }
    WSTEP(cudaMemcpyAsync(idx, flag, sizeof(uint32_t) * nint, cudaMemcpyDeviceToDevice, st));
    k_scan<<<1, 1024, 0, st>>>(idx, nint);
    WSTEP(cudaGetLastError());
    {
        uint32_t last_idx = 0, last_flag = 0;
        WSTEP(cudaMemcpyAsync(&last_idx, idx + nint - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        WSTEP(cudaMemcpyAsync(&last_flag, flag + nint - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        WSTEP(cudaStreamSynchronize(st));
        nwide = last_idx + last_flag;
    }
    WSTEP(cudaMalloc(&S->wide, sizeof(float4) * kWideF4 * (size_t)nwide));
    WSTEP(cudaMalloc(&S->wide_src, sizeof(int32_t) * kWideChildren * (size_t)nwide));
    S->nwide = nwide;
    S->bytes += sizeof(float4) * kWideF4 * (size_t)nwide + sizeof(int32_t) * kWideChildren * (size_t)nwide;
    k_wide_write<<<cdiv(nint, 128), 128, 0, st>>>(S->nodes, S->trav, n, flag, idx, S->wide, S->wide_src);
    WSTEP(cudaGetLastError());
    WSTEP(cudaStreamSynchronize(st));
#undef WSTEP
wdone:
    cudaFree(flag);
    cudaFree(idx);
    cudaFree(cnt);
    cudaFree(fa);
    cudaFree(fb);
    return rc;
}

// A scene's buffers are one allocation (cudaMalloc and cudaFree wait for the
// device: 14 and 7 of them took longer than a small build), and the build's
// scratch lies in it: the sort's buffers where the nodes go, uploaded spheres
// where the traversal records go.
venu_status build_scene(const venu_sphere* spheres, bool on_host, uint32_t n, cudaStream_t st, venu_scene* S) {
    S->n = n;
    if (n == 0) return VENU_OK;
    if (n > (1u << 28)) {
        set_error("venu_scene_create: more than 2^28 spheres");
        return VENU_ERR_TOO_LARGE;
    }
    const size_t N = n, nint = n > 1 ? n - 1 : 1;
    const bool general = n > kSmallScene;  // the radix sort, not the one-block path
    const size_t hist_b = general ? al256(sizeof(uint32_t) * kBuckets * (size_t)cdiv(n, 32 * sort_rounds(n))) : 0;
    const size_t words_b = al256(sizeof(uint32_t) * N);
    const size_t sort_b = general ? 3 * words_b + hist_b + al256(sizeof(uint32_t) * 4 * kBuckets) : words_b;
    const size_t nodes_b = al256(std::max(sizeof(float4) * 2 * nint, sort_b));
    const size_t trav_b = al256(std::max(sizeof(float4) * (4 * nint + 3), sizeof(venu_sphere) * N));
    const size_t sph_b = al256(sizeof(float4) * N), par_b = al256(sizeof(int32_t) * (nint + N));
    const size_t arr_b = al256(sizeof(uint32_t) * nint), ctl_b = al256(sizeof(LbvhCtl));
    const size_t err_b = al256(sizeof(uint32_t) * kTraceWords);
    const size_t total = nodes_b + trav_b + 2 * sph_b + 2 * words_b + par_b + arr_b + ctl_b + err_b;
    VENU_CUDA(cudaMalloc(&S->arena, total));
    S->bytes = total;
    unsigned char* at = static_cast<unsigned char*>(S->arena);
    auto take = [&](size_t b) {
        unsigned char* p = at;
        at += b;
        return p;
    };
    unsigned char* const scratch = take(nodes_b);
    S->nodes = reinterpret_cast<float4*>(scratch);
    S->trav = reinterpret_cast<float4*>(take(trav_b));
    S->sph = reinterpret_cast<float4*>(take(sph_b));
    S->mat = reinterpret_cast<float4*>(take(sph_b));
    S->meta = reinterpret_cast<uint32_t*>(take(words_b));
    S->keys = reinterpret_cast<uint32_t*>(take(words_b));
    S->parents = reinterpret_cast<int32_t*>(take(par_b));
    S->arrive = reinterpret_cast<uint32_t*>(take(arr_b));
    LbvhBuffers B{};
    B.ctl = reinterpret_cast<LbvhCtl*>(take(ctl_b));
    S->trace_err = reinterpret_cast<uint32_t*>(take(err_b));
    B.nodes = S->nodes;
    B.trav = S->trav;
    B.sph = S->sph;
    B.mat = S->mat;
    B.meta = S->meta;
    B.keys = S->keys;
    B.pint = S->parents;
    B.pleaf = S->parents + nint;
    B.arrive = S->arrive;
    B.trace_err = S->trace_err;
    B.vals = reinterpret_cast<uint32_t*>(scratch);
    if (general) {
        B.keys_alt = reinterpret_cast<uint32_t*>(scratch + words_b);
        B.vals_alt = reinterpret_cast<uint32_t*>(scratch + 2 * words_b);
        B.hist = reinterpret_cast<uint32_t*>(scratch + 3 * words_b);
        B.totals = reinterpret_cast<uint32_t*>(scratch + 3 * words_b + hist_b);
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    venu_status rc = VENU_OK;
    LbvhCtl hc;
#define STEP(call)                               \
    do {                                         \
        cudaError_t _e = (call);                 \
        if (_e != cudaSuccess) {                 \
            rc = cuda_fail(_e, #call);           \
            goto done;                           \
        }                                        \
    } while (0)
    if (on_host) {
        STEP(cudaMemcpyAsync(S->trav, spheres, sizeof(venu_sphere) * N, cudaMemcpyHostToDevice, st));
        spheres = reinterpret_cast<const venu_sphere*>(S->trav);
    }
    STEP(cudaEventCreate(&e0));
    STEP(cudaEventCreate(&e1));
    STEP(cudaEventRecord(e0, st));
    STEP(launch_lbvh(spheres, n, st, B));
    STEP(cudaEventRecord(e1, st));
    STEP(cudaMemcpyAsync(&hc, B.ctl, sizeof(LbvhCtl), cudaMemcpyDeviceToHost, st));
    STEP(cudaStreamSynchronize(st));
    {
        float ms = 0.0f;
        STEP(cudaEventElapsedTime(&ms, e0, e1));
        S->build_ms = ms;
        std::memcpy(S->bounds, hc.bounds, sizeof(S->bounds));
        S->nhoist = n > 1 ? hc.hoisted.n : 0u;
        for (int i = 0; i < kMaxHoisted; ++i) S->hoist[i] = hc.hoisted.slot[i];
        if (n > 1 && hc.bad_words) {
            set_error("venu_scene_create: the LBVH build produced " + std::to_string(hc.bad_words) +
                      " out-of-range child words");
            rc = VENU_ERR_INVALID;
        }
    }
#undef STEP
done:
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (rc != VENU_OK) cudaStreamSynchronize(st);  // nothing may still write to what the caller frees
    return rc;
}

venu_status ensure_wide(const venu_scene* S, cudaStream_t st) {
    std::lock_guard<std::mutex> lock(S->wide_mu);
    if (S->n < 2 || S->wide) return VENU_OK;
    const auto t0 = std::chrono::steady_clock::now();
    // after the refits called for so far, and before any that is called for from
    // now on: those find the whole tree and refit it, too
    std::lock_guard<std::mutex> refits(S->refit_mu);
    if (S->refit_done) VENU_CUDA(cudaStreamWaitEvent(st, S->refit_done, 0));
    const venu_status rc = build_wide(S, st);
    S->wide_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - t0).count();
    if (rc != VENU_OK) {  // no half-built tree stays behind
        cudaStreamSynchronize(st);
        cudaFree(S->wide);
        cudaFree(S->wide_src);
        if (S->nwide)
            S->bytes -= sizeof(float4) * kWideF4 * (size_t)S->nwide + sizeof(int32_t) * kWideChildren * (size_t)S->nwide;
        S->wide = nullptr;
        S->wide_src = nullptr;
        S->nwide = 0;
    }
    return rc;
}

namespace {
// The refit's launches, with its n - 1 arrival counters.
cudaError_t launch_refit(venu_scene* S, const venu_sphere* s, uint32_t* arrive, cudaStream_t st) {
    const uint32_t n = S->n;
    k_gather<<<cdiv(n, 256), 256, 0, st>>>(s, S->meta, 0x3fffffffu, n, S->sph, S->mat, S->meta, nullptr, arrive);
    if (n == 1) return cudaGetLastError();
    k_refit<<<cdiv(n, 256), 256, 0, st>>>(S->sph, (int)n, S->nodes, S->parents, S->parents + (n - 1), arrive);
    HoistList list{S->nhoist, {}};
    for (int i = 0; i < kMaxHoisted; ++i) list.slot[i] = S->hoist[i];
    const cudaError_t e = launch_trav_layout(S->nodes, S->sph, n, S->trav, S->parents, S->parents + (n - 1), nullptr, list,
                                             nullptr, st);
    if (e != cudaSuccess) return e;
    if (S->nwide) k_wide_refit<<<cdiv(S->nwide, 128), 128, 0, st>>>(S->trav, S->nwide, S->wide_src, S->wide);
    return cudaGetLastError();
}
}  // namespace

// New sphere records into the same slots (meta holds each slot's original
// index), then the boxes bottom-up over the kept parent links, then the
// traversal records.  Topology, slot order and the hoisted set stay those of the
// build.
//
// The arrival counters are the build's (two stream-ordered allocations took
// 180 us a call), cleared by each refit, and refits of one scene run one after
// another: two that overlapped would count each other's arrivals and make boxes
// from children that are not there yet.  A captured refit, which can replay
// beside any other, brings counters of its own into the graph.
venu_status update_scene(venu_scene* S, const venu_sphere* s, bool on_host, cudaStream_t st) {
    const uint32_t n = S->n;
    if (n == 0) return VENU_OK;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    VENU_CUDA(cudaStreamIsCapturing(st, &capture));
    const bool captured = capture != cudaStreamCaptureStatusNone;
    std::lock_guard<std::mutex> lock(S->refit_mu);
    if (!captured) {
        if (S->refit_done) VENU_CUDA(cudaStreamWaitEvent(st, S->refit_done, 0));
        else VENU_CUDA(cudaEventCreateWithFlags(&S->refit_done, cudaEventDisableTiming));
    }
    if (on_host) {  // a failed upload leaves the scene as it was
        const size_t bytes = sizeof(venu_sphere) * (size_t)n;
        if (!S->upload) {
            VENU_CUDA(cudaMalloc(&S->upload, bytes));
            S->bytes += bytes;
        }
        VENU_CUDA(cudaMemcpyAsync(S->upload, s, bytes, cudaMemcpyHostToDevice, st));
        s = S->upload;
    }
    uint32_t* arrive = S->arrive;
    if (captured && n > 1) VENU_CUDA(cudaMallocAsync(&arrive, sizeof(uint32_t) * (n - 1), st));
    cudaError_t e = launch_refit(S, s, arrive, st);
    const cudaError_t end = !captured ? cudaEventRecord(S->refit_done, st) : n > 1 ? cudaFreeAsync(arrive, st) : cudaSuccess;
    if (e == cudaSuccess) e = end;
    return e == cudaSuccess ? VENU_OK : cuda_fail(e, "venu_scene_update");
}

}  // namespace venu

// ---------------------------------------------------------------------------
// venu_lbvh_build_noalloc: the same LBVH build into caller-owned buffers,
// with its scratch in a fixed file-scope device array instead of cudaMalloc.
// ---------------------------------------------------------------------------
namespace venu {
namespace {

constexpr uint32_t kNoAllocMaxSpheres = VENU_NOALLOC_MAX_SPHERES;
constexpr uint32_t kNoAllocMaxTiles = (kNoAllocMaxSpheres + 127) / 128;  // sort_rounds: 128 keys a tile
static_assert(kNoAllocMaxSpheres <= 65536, "sort_rounds gives tiles of 128 keys up to 65536 spheres");
constexpr size_t kNA = kNoAllocMaxSpheres;
constexpr size_t kOffCtl = 0;                                         // LbvhCtl
constexpr size_t kOffKeysAlt = al256(kOffCtl + sizeof(LbvhCtl));
constexpr size_t kOffVals = al256(kOffKeysAlt + 4 * kNA);
constexpr size_t kOffValsAlt = al256(kOffVals + 4 * kNA);
constexpr size_t kOffHist = al256(kOffValsAlt + 4 * kNA);
constexpr size_t kOffTotals = al256(kOffHist + 4 * (size_t)kBuckets * kNoAllocMaxTiles);
constexpr size_t kOffArrive = al256(kOffTotals + 4 * 4 * (size_t)kBuckets);
constexpr size_t kOffParentInt = al256(kOffArrive + 4 * kNA);
constexpr size_t kOffParentLeaf = al256(kOffParentInt + 4 * kNA);
constexpr size_t kNoAllocScratchBytes = al256(kOffParentLeaf + 4 * kNA);  // about 2.1 MB

}  // namespace
}  // namespace venu

// Every GPU that loads the library holds this array until the process exits.
static __device__ __align__(256) unsigned char g_lbvh_noalloc_scratch[venu::kNoAllocScratchBytes];

namespace venu {
namespace {

std::mutex g_noalloc_mu;
constexpr int kMaxDevices = 64;
void* g_noalloc_scratch[kMaxDevices] = {};

// Device address of the scratch array on the current device.  The host-side
// name g_lbvh_noalloc_scratch is only a stand-in: its device address comes
// from cudaGetSymbolAddress, once per device, with that device current.
venu_status noalloc_scratch(unsigned char** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "venu_lbvh_build_noalloc: cudaGetDevice");
    if (dev < 0 || dev >= kMaxDevices) {
        set_error("venu_lbvh_build_noalloc: device ordinal out of range");
        return VENU_ERR_INVALID;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_scratch[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_lbvh_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "venu_lbvh_build_noalloc: cudaGetSymbolAddress");
        g_noalloc_scratch[dev] = p;
    }
    *out = static_cast<unsigned char*>(g_noalloc_scratch[dev]);
    return VENU_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace
}  // namespace venu

extern "C" venu_status venu_lbvh_build_noalloc(const venu_sphere* spheres_dev, uint32_t n, float* nodes_out,
                                               float* spheres_out, float* materials_out, uint32_t* meta_out,
                                               uint32_t* morton_out, void* stream) {
    using namespace venu;
    if (n > kNoAllocMaxSpheres) {
        set_error("venu_lbvh_build_noalloc: " + std::to_string(n) + " spheres exceed the limit of " +
                  std::to_string(kNoAllocMaxSpheres) + " (VENU_NOALLOC_MAX_SPHERES); use venu_scene_create");
        return VENU_ERR_TOO_LARGE;
    }
    if (n == 0) return VENU_OK;
    if (!spheres_dev || !spheres_out || !materials_out || !meta_out || !morton_out || (n > 1 && !nodes_out)) {
        set_error("venu_lbvh_build_noalloc: NULL buffer");
        return VENU_ERR_INVALID;
    }
    if (!aligned16(spheres_out) || !aligned16(materials_out) || (n > 1 && !aligned16(nodes_out))) {
        set_error("venu_lbvh_build_noalloc: nodes/spheres/materials outputs must be 16-byte aligned");
        return VENU_ERR_INVALID;
    }
    venu_status ds = require_device();
    if (ds != VENU_OK) return ds;
    unsigned char* base = nullptr;
    venu_status ss = noalloc_scratch(&base);
    if (ss != VENU_OK) return ss;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    LbvhBuffers B{};
    B.nodes = reinterpret_cast<float4*>(nodes_out);
    B.sph = reinterpret_cast<float4*>(spheres_out);
    B.mat = reinterpret_cast<float4*>(materials_out);
    B.meta = meta_out;
    B.keys = morton_out;
    B.ctl = reinterpret_cast<LbvhCtl*>(base + kOffCtl);
    B.keys_alt = reinterpret_cast<uint32_t*>(base + kOffKeysAlt);
    B.vals = reinterpret_cast<uint32_t*>(base + kOffVals);
    B.vals_alt = reinterpret_cast<uint32_t*>(base + kOffValsAlt);
    B.hist = reinterpret_cast<uint32_t*>(base + kOffHist);
    B.arrive = reinterpret_cast<uint32_t*>(base + kOffArrive);
    B.pint = reinterpret_cast<int32_t*>(base + kOffParentInt);
    B.pleaf = reinterpret_cast<int32_t*>(base + kOffParentLeaf);
    B.totals = reinterpret_cast<uint32_t*>(base + kOffTotals);
    // The scratch keeps the previous call's contents; launch_lbvh resets what
    // must start from a known value (bounds seeds, hoist counters, arrival
    // counters, parent links) before using it.
    VENU_CUDA(launch_lbvh(spheres_dev, n, st, B));
    VENU_CUDA(cudaGetLastError());
    return VENU_OK;
}
