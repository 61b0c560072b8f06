// venu_device.cuh -- device building blocks of the GB300 path tracer.
//
// Arithmetic contract (the library is compiled with -fmad=false): every
// float operation rounds once as written; fmaf() appears only where written.
// Camera rays, scattering and the sky follow the reference's device source
// (Core/RayTracer.cu, Core/vec_math.h) operation by operation; the ray/box
// and ray/sphere tests are this library's own (robust slab test, stable
// quadratic with an exactly refined constant term).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/venu.h"

#ifndef VENU_MINMAX3
#define VENU_MINMAX3 1
#endif
// Register caps of the binary tree's kernels.  The bounce kernel: at 56 nine
// blocks of 128 threads (36 warps) stay resident per SM (1080p x 32 RTIOW at 48 /
// 56 / 64 / 72: 13.53 / 13.23 / 13.36 / 14.28 ms).  The finishing kernel: 64 (400x225
// x 16 at 48 / 56 / 64: 588 / 562 / 559 us; 300k spheres gain 1.6 % at 56, the
// 4-wide tree loses 4 %).  The walk of large bounces: 64 (1M spheres 1080p x 4 at
// 56 / 64 / 72: 72.1 / 71.2 / 79.2 ms).
#ifndef VENU_TRACE_MAXREG
#define VENU_TRACE_MAXREG 56
#endif
#define VENU_TRACE_BOUNDS __maxnreg__(VENU_TRACE_MAXREG)
#ifndef VENU_FINISH_MAXREG
#define VENU_FINISH_MAXREG 64
#endif
#define VENU_FINISH_BOUNDS __maxnreg__(VENU_FINISH_MAXREG)
#ifndef VENU_WALK_MAXREG
#define VENU_WALK_MAXREG 64
#endif
#define VENU_WALK_BOUNDS __maxnreg__(VENU_WALK_MAXREG)
// Register cap of the fused kernel over the wide tree.  With 4 children per
// node, 64 registers (8 resident 128-thread blocks per SM, a few spilled
// bytes) beat 72 and 80 (6 and 5 blocks) on RTIOW (+5 %) and 1M spheres
// (+7 %), and lose 3 % on 5k spheres.
#ifndef VENU_WIDE_MAXREG
#define VENU_WIDE_MAXREG 64
#endif
#define VENU_WIDE_BOUNDS __maxnreg__(VENU_WIDE_MAXREG)
// The batch engine's kernels (96 uneven jobs at 56 / 64 / 72: 6.66 / 6.54 / 7.16 ms).
#ifndef VENU_TRACE_MULTI_MAXREG
#define VENU_TRACE_MULTI_MAXREG 64
#endif
#define VENU_TRACE_MULTI_BOUNDS __maxnreg__(VENU_TRACE_MULTI_MAXREG)

namespace venu {

// ---------------------------------------------------------------------------
// float3 operations with Core/vec_math.h semantics.
// ---------------------------------------------------------------------------
struct f3 {
    float x, y, z;
};
__device__ __forceinline__ f3 mk(float x, float y, float z) { return f3{x, y, z}; }
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ f3 operator-(f3 a) { return mk(-a.x, -a.y, -a.z); }
__device__ __forceinline__ f3 operator*(f3 a, f3 b) { return mk(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ f3 operator*(float s, f3 a) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
// Core/vec_math.h:483-487: float3 / float multiplies by the reciprocal.
__device__ __forceinline__ f3 divs(f3 a, float s) {
    float inv = 1.0f / s;
    return a * inv;
}
__device__ __forceinline__ f3 normalize(f3 v) {  // Core/vec_math.h:544-549
    float inv = 1.0f / sqrtf(dot(v, v));
    return v * inv;
}
__device__ __forceinline__ f3 reflect(f3 i, f3 n) { return i - (2.0f * n) * dot(n, i); }
__device__ __forceinline__ f3 refract(f3 uv, f3 n, float eta) {  // Core/vec_math.h:563-569
    float cos_theta = fminf(dot(-uv, n), 1.0f);
    f3 r_perp = eta * (uv + cos_theta * n);
    f3 r_par = (-sqrtf(fabsf(1.0f - dot(r_perp, r_perp)))) * n;
    return r_perp + r_par;
}
__device__ __forceinline__ f3 lerp3(f3 a, f3 b, float t) { return a + t * (b - a); }

// ---------------------------------------------------------------------------
// RNG: TEA-4 seed hash and the 24-bit LCG of Core/random.cuh:31-67.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tea4(uint32_t v0, uint32_t v1) {
    uint32_t s0 = 0;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        s0 += 0x9e3779b9u;
        v0 += ((v1 << 4) + 0xa341316cu) ^ (v1 + s0) ^ ((v1 >> 5) + 0xc8013ea4u);
        v1 += ((v0 << 4) + 0xad90777du) ^ (v0 + s0) ^ ((v0 >> 5) + 0x7e95761eu);
    }
    return v0;
}
__device__ __forceinline__ float rnd(uint32_t& s) {
    s = 1664525u * s + 1013904223u;
    return (float)(s & 0x00FFFFFFu) / (float)0x01000000;
}
// Core/RayTracer.cu:93-97 with min=-1, max=1; draws x, y, z left to right.
// The rejection loops stop after kMaxTries candidates (the last one is then
// kept): an acceptance rate of 52% (sphere) / 79% (disk) makes that bound
// unreachable in practice, and it guarantees termination on the GPU.
constexpr int kMaxTries = 4096;
// -1 + 2 rnd(s): both products are by powers of two and the sum is a multiple
// of 2^-23 in [-1, 1), so one fmaf of the 24-bit integer gives the same float.
__device__ __forceinline__ float rnd_pm1(uint32_t& s) {
    s = 1664525u * s + 1013904223u;
    return fmaf((float)(s & 0x00FFFFFFu), 1.1920928955078125e-07f, -1.0f);  // 2^-23
}
__device__ __forceinline__ f3 random_in_unit_sphere(uint32_t& s) {  // :117-125
    f3 p;
    for (int i = 0; i < kMaxTries; ++i) {
        float x = rnd_pm1(s);
        float y = rnd_pm1(s);
        float z = rnd_pm1(s);
        p = mk(x, y, z);
        if (!(dot(p, p) >= 1.0f)) break;
    }
    return p;
}
__device__ __forceinline__ f3 random_in_unit_disk(uint32_t& s) {  // :141-149
    f3 p;
    for (int i = 0; i < kMaxTries; ++i) {
        float x = rnd_pm1(s);
        float y = rnd_pm1(s);
        p = mk(x, y, 0.0f);
        if (!(dot(p, p) >= 1.0f)) break;
    }
    return p;
}
// Core/RayTracer.cu:8-13; for float x, (double)x < 1e-8 <=> x <= 1e-8f.
__device__ __forceinline__ bool near_zero(f3 e) {
    return fabsf(e.x) <= 1e-8f && fabsf(e.y) <= 1e-8f && fabsf(e.z) <= 1e-8f;
}

// ---------------------------------------------------------------------------
// Camera (Params fields) with the per-launch constants normalize(U/V).
// ---------------------------------------------------------------------------
struct DevCamera {
    f3 origin, u, v, w, un, vn;
    float lens;
};

// Core/RayTracer.cu:151-161,173-177: jitter u, jitter v, then the lens disk.
__device__ __forceinline__ void camera_ray(const DevCamera& C, uint32_t x, uint32_t y, uint32_t W,
                                           uint32_t H, uint32_t& seed, f3& o, f3& d) {
    float r1 = rnd(seed);
    float s = 2.0f * ((float)x + r1) / (float)(W - 1) - 1.0f;
    float r2 = rnd(seed);
    float t = 2.0f * ((float)y + r2) / (float)(H - 1) - 1.0f;
    f3 rd = C.lens * random_in_unit_disk(seed);
    f3 offset = C.un * rd.x + C.vn * rd.y;
    o = C.origin + offset;
    d = C.w + (s * C.u) * 0.5f + (t * C.v) * 0.5f - offset;
}

// Core/RayTracer.cu:442-449.  fmaf(0.5, y, 0.5) equals the reference's double
// 0.5 * (y + 1.0) rounded to float (both are one rounding of the same value).
__device__ __forceinline__ f3 sky(f3 d) {
    f3 ud = normalize(d);
    float t = fmaf(0.5f, ud.y, 0.5f);
    return lerp3(mk(1.0f, 1.0f, 1.0f), mk(0.5f, 0.7f, 1.0f), t);
}

// Schlick (Core/RayTracer.cu:373-379) with (1-cos)^5 as an explicit product.
__device__ __forceinline__ float reflectance(float cosine, float ref_idx) {
    float r0 = (1.0f - ref_idx) / (1.0f + ref_idx);
    r0 = r0 * r0;
    float x = 1.0f - cosine;
    float x2 = x * x;
    float x5 = (x2 * x2) * x;
    return r0 + (1.0f - r0) * x5;
}

// x^(1/2.4) for x in [2^-126, 1], the power of the sRGB encode
// (Core/RayTracer.cu:16-47 calls powf), from IEEE +, -, *, / and fmaf only,
// so that the host restatement rounds identically and image bytes can be
// checked exactly.  x = m 2^e with m in [sqrt(1/2), sqrt(2));
// log2 m = s (c1 + c3 s^2 + c5 s^4 + c7 s^6 + c9 s^8), s = (m-1)/(m+1): the
// atanh series of ln m = 2 atanh(s) scaled by 1/ln 2 (c_k = 2/(k ln 2), c1
// as a head and a tail); t = y (e + log2 m) with the product y e split
// exactly (TwoProduct); 2^t = 2^n 2^f with n = rint(t) and 2^f by its Taylor
// series to f^7 (coefficients ln(2)^k / k!).  Error at most 1.16 ulp over
// every float in [0.0031308, 1] (measured against double pow).
__device__ __forceinline__ float srgb_pow(float x) {
    const uint32_t b = __float_as_uint(x);
    int e = (int)(b >> 23) - 127;
    float m = __uint_as_float((b & 0x007fffffu) | 0x3f800000u);
    if (m > 1.41421353816986083984375f) {
        m = m * 0.5f;
        e += 1;
    }
    const float s = (m - 1.0f) / (m + 1.0f);
    const float z = s * s;
    float tail = fmaf(z, 0.32059890031814575f, 0.41219857335090637f);
    tail = fmaf(z, tail, 0.5770780444145203f);
    tail = fmaf(z, tail, 0.9617967009544373f);
    tail = fmaf(z, tail, 3.8519259e-08f);
    const float L = fmaf(s, 2.885390043258667f, s * tail);
    const float y = 0.4166666567325592f;  // 1.0f / 2.4f, the reference's exponent
    const float fe = (float)e;
    const float ph = fe * y;
    const float pl = fmaf(fe, y, -ph);
    const float q = fmaf(y, L, pl);
    const float n = rintf(ph + q);
    const float f = (ph - n) + q;
    float p = fmaf(f, 1.5252733646775596e-05f, 1.540352968731895e-04f);
    p = fmaf(f, p, 1.3333557872101665e-03f);
    p = fmaf(f, p, 9.618128649890423e-03f);
    p = fmaf(f, p, 5.550410971045494e-02f);
    p = fmaf(f, p, 2.4022650718688965e-01f);
    p = fmaf(f, p, 6.931471824645996e-01f);
    p = fmaf(f, p, 1.0f);
    return p * __uint_as_float((uint32_t)(127 + (int)n) << 23);
}

// ---------------------------------------------------------------------------
// Scene view: LBVH nodes + spheres/materials in Morton (slot) order.
// ---------------------------------------------------------------------------
// Child words: bit 31 = leaf, bit 30 = leaf already tested before the
// traversal (a hoisted huge sphere), bits 0-29 = slot or internal index.
constexpr int32_t kLeaf = (int32_t)0x80000000u;
constexpr int32_t kHoisted = 0x40000000;
constexpr int32_t kSlotMask = 0x3fffffff;
constexpr int32_t kNone = 0x7fffffff;
constexpr int kMaxHoisted = 4;

// Children per node of the wide traversal tree (4; 8 measured slower on every
// workload here) and its float4s: centres and half extents of the four
// children's boxes per axis at 2a and 2a + 1, then the child words at 6.
constexpr int kWideW = 4;
constexpr int kWideF4 = 8;

struct SceneView {
    const float4* __restrict__ nodes;  // 2 float4 per internal node: {lo, left} {hi, right}
    const float4* __restrict__ trav;   // 4 float4 per internal node: both children, see lbvh.cu
    const float4* __restrict__ wide;   // kWideF4 float4 per node of the wide tree, see lbvh.cu
    const float4* __restrict__ sph;    // {center, radius} per slot
    const float4* __restrict__ mat;    // {albedo, fuzz or ir} per slot
    const uint32_t* __restrict__ meta; // original id | material << 30
    uint32_t n;
    uint32_t nhoist;                   // huge spheres tested first by every ray
    int32_t hoist[kMaxHoisted];        // their slots (ascending)
};

// A scene by its entry in a job table (the batch engine): only the record
// pointer is held in registers through a walk, the rest is read where it is
// needed, through L1 (96 uneven jobs 6.65 -> 6.55 ms against a whole SceneView a
// lane; with volatile reads, which pass L1 by, 7.86).
struct JobScene {
    const float4* __restrict__ trav;
    const SceneView* g;
};
__device__ __forceinline__ const float4* sv_sph(const SceneView& S) { return S.sph; }
__device__ __forceinline__ const float4* sv_sph(const JobScene& S) { return S.g->sph; }
__device__ __forceinline__ const float4* sv_nodes(const SceneView& S) { return S.nodes; }
__device__ __forceinline__ const float4* sv_nodes(const JobScene& S) { return S.g->nodes; }
__device__ __forceinline__ uint32_t sv_n(const SceneView& S) { return S.n; }
__device__ __forceinline__ uint32_t sv_n(const JobScene& S) { return S.g->n; }
__device__ __forceinline__ uint32_t sv_nhoist(const SceneView& S) { return S.nhoist; }
__device__ __forceinline__ uint32_t sv_nhoist(const JobScene& S) { return S.g->nhoist; }
__device__ __forceinline__ int32_t sv_hoist(const SceneView& S, int h) { return S.hoist[h]; }
__device__ __forceinline__ int32_t sv_hoist(const JobScene& S, int h) { return S.g->hoist[h]; }

// Slab test: a box's entry / exit parameter on axis k is
// fma(lo_k or hi_k, inv_k, offset).  The offset -(o_k inv_k) is rounded, which
// a margin of |o_k inv_k| 2^-21 covers (several times that rounding).
//   Shared margin (almost every ray): one offset n0_k = -(o_k inv_k) per axis
//   and the largest margin of the three axes added once to the exit
//   parameter (n1.x), which keeps four floats live during traversal.
//   Per-axis margins (axis = true): a near-zero direction component (1/d up
//   to 1e20) makes its own margin huge, and shared by all axes it would
//   switch off the culling on the other two (such a ray then visits every
//   node its slab meets).  When the shared margin exceeds 1 (in units of t)
//   the offsets carry each axis's own margin instead, moved outwards: n0_k
//   for the lo plane, n1_k for the hi plane (the entry plane is lo when
//   inv_k >= 0).  Such rays are rare (a direction component below ~1e-5 of
//   the others) and traverse with their own instantiation of the loop.
//   from: slot of the sphere the ray leaves (its origin lies on that
//   sphere's surface), or -1 (camera rays, rays from the caller).
//   m: what the fast walk adds to exit parameters (far_margin).
struct RayPre {
    f3 o, d, inv, n0, n1;
    float a, inv_a, m;
    bool axis;
    int32_t from;
};

constexpr float kSharedMarginMax = 1.0f;

// The same ray with per-axis margins (for the canonical walk's AXIS form).
__device__ __forceinline__ void axis_margins(RayPre& R) {
    const float px = R.o.x * R.inv.x, py = R.o.y * R.inv.y, pz = R.o.z * R.inv.z;
    const float mx = fabsf(px) * 4.76837158203125e-07f;  // 2^-21
    const float my = fabsf(py) * 4.76837158203125e-07f;
    const float mz = fabsf(pz) * 4.76837158203125e-07f;
    const float lx = -px - mx, hx = -px + mx;
    const float ly = -py - my, hy = -py + my;
    const float lz = -pz - mz, hz = -pz + mz;
    R.n0 = mk(R.inv.x >= 0.0f ? lx : hx, R.inv.y >= 0.0f ? ly : hy, R.inv.z >= 0.0f ? lz : hz);
    R.n1 = mk(R.inv.x >= 0.0f ? hx : lx, R.inv.y >= 0.0f ? hy : ly, R.inv.z >= 0.0f ? hz : lz);
    R.axis = true;
}

// 1/x by the hardware approximation (one ulp), for x not subnormal.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// APPROX: 1/d good to an ulp, which is all the fast walk asks of it: it serves
// the slab tests alone, whose margins count the ulp, and no hit depends on it (1/a
// below enters the hits and stays correctly rounded).  Correctly rounded: RTIOW
// 1920x1080 x 256 +0.8 %, 1200x800 x 16 +1.6 %, 96 uneven jobs +0.7 %, images the
// same.
template <bool APPROX>
__device__ __forceinline__ RayPre prep(f3 o, f3 d) {
    RayPre R;
    R.from = -1;
    R.m = 0.0f;
    R.o = o;
    R.d = d;
    float dx = fabsf(d.x) < 1e-20f ? copysignf(1e-20f, d.x) : d.x;
    float dy = fabsf(d.y) < 1e-20f ? copysignf(1e-20f, d.y) : d.y;
    float dz = fabsf(d.z) < 1e-20f ? copysignf(1e-20f, d.z) : d.z;
    R.inv = APPROX ? mk(rcp_approx(dx), rcp_approx(dy), rcp_approx(dz)) : mk(1.0f / dx, 1.0f / dy, 1.0f / dz);
    const float px = o.x * R.inv.x, py = o.y * R.inv.y, pz = o.z * R.inv.z;
    const float mx = fabsf(px) * 4.76837158203125e-07f;  // 2^-21
    const float my = fabsf(py) * 4.76837158203125e-07f;
    const float mz = fabsf(pz) * 4.76837158203125e-07f;
    const float m = fmaxf(fmaxf(mx, my), mz);
    R.axis = m > kSharedMarginMax;
    R.n0 = mk(-px, -py, -pz);
    R.n1 = mk(m, 0.0f, 0.0f);
    R.a = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));
    R.inv_a = 1.0f / R.a;
    return R;
}

// Three-input min / max (one instruction on sm_100 and later).  The slab
// test never feeds them a NaN (the direction guard keeps 1/d finite), and on
// non-NaN inputs they equal the two-input chains exactly.
__device__ __forceinline__ float fmax3(float a, float b, float c) {
#if VENU_MINMAX3
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
#if VENU_MINMAX3
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fminf(fminf(a, b), c);
#endif
}

// Robust slab test: conservative by a relative 2^-20 plus the rounding
// margins of the slab offsets (shared or per axis, see RayPre), so rounding
// never drops a box the ray touches.
template <bool AXIS>
__device__ __forceinline__ bool box_test(const RayPre& R, float4 lo, float4 hi, float tmin,
                                         float tcap, float& tnear) {
    const f3 nh = AXIS ? R.n1 : R.n0;
    float t0x = fmaf(lo.x, R.inv.x, R.n0.x), t1x = fmaf(hi.x, R.inv.x, nh.x);
    float t0y = fmaf(lo.y, R.inv.y, R.n0.y), t1y = fmaf(hi.y, R.inv.y, nh.y);
    float t0z = fmaf(lo.z, R.inv.z, R.n0.z), t1z = fmaf(hi.z, R.inv.z, nh.z);
    float tn = fmax3(fminf(t0x, t1x), fminf(t0y, t1y), fmaxf(fminf(t0z, t1z), tmin));
    float tf = fmin3(fmaxf(t0x, t1x), fmaxf(t0y, t1y), fminf(fmaxf(t0z, t1z), tcap));
    tnear = tn;
    // tf (1 + 2^-20) covers the roundings of the two fmas; the shared margin
    // is added here
    return AXIS ? tn <= tf * 1.00000095367431640625f : tn <= fmaf(tf, 1.00000095367431640625f, R.n1.x);
}

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    float bp = s - a;
    float ap = s - bp;
    e = (a - ap) + (b - bp);
}

// Two floats in one 64-bit register pair, and the packed FMA of sm_100 and
// later (each half is one ordinary fmaf).
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Packed sum and product; fma2(b, neg1, a) is a - b (one rounding).
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// 32 bytes with one instruction (32-byte aligned, read-only data).
__device__ __forceinline__ void ldg32(const void* p, f2& a, f2& b, f2& c, f2& d) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// Ray/sphere: the discriminant is formed from the perpendicular distance of
// the centre to the ray line, disc = a (r^2 - |f|^2) with f = h - (h.d/a) d
// (Haines et al., "Precision Improvements for Ray/Sphere Intersection", Ray
// Tracing Gems ch. 7), so its error scales with r^2 instead of |h|^2; the
// roots come from q = -(b + sign(b) sqrt(disc)) as q/a and c/q (no
// cancellation).  When the origin is close to the surface relative to the
// radius (|c| < (|h|^2 + r^2)/16), c = |o-C|^2 - r^2 and h are refined with
// TwoDiff/TwoProduct/TwoSum error terms (x and y packed; packing the second half
// of the branch as well loses again what this gains: RTIOW 1920x1080 x 32 13.10
// -> 12.95 ms, 13.07 with both), so the near root c/q keeps full relative accuracy
// even for the r = 1000 ground sphere.  Root selection
// follows Core/RayTracer.cu:248-253: the smaller root in [tmin, tmax], else
// the larger.
__device__ __forceinline__ bool sphere_test(const RayPre& R, float4 S, float tmin, float tmax,
                                            float& tout) {
    const float r = S.w;
    float hx = R.o.x - S.x, hy = R.o.y - S.y, hz = R.o.z - S.z;
    float hb = fmaf(hx, R.d.x, fmaf(hy, R.d.y, hz * R.d.z));
    float hh = fmaf(hx, hx, fmaf(hy, hy, hz * hz));
    float r2 = r * r;
    float c = hh - r2;
    // Origin clearly outside (c above its rounding bound) and moving away from
    // the centre (h.d > 0): both roots are negative, no hit.
    if (hb > 0.0f && c > (hh + r2) * 9.5367431640625e-07f) return false;  // 2^-20
    float discp;
    const f2 neg1 = pack2(-1.0f, -1.0f);
    if (fabsf(c) < (hh + r2) * 0.0625f) {
        // exact residuals of h = o - C (TwoDiff)
        const f2 O = pack2(R.o.x, R.o.y), Cn = pack2(-S.x, -S.y), H = pack2(hx, hy);
        const f2 Bv = fma2(H, neg1, O);
        const f2 E2 = add2(fma2(add2(H, Bv), neg1, O), add2(Bv, Cn));
        float bvz = R.o.z - hz;
        float ex, ey;
        unpack2(E2, ex, ey);
        float ez = (R.o.z - (hz + bvz)) + (bvz - S.z);
        // c = |h + e|^2 - r^2 from exact squares and compensated sums
        const f2 P2 = mul2(H, H);
        const f2 Q2 = fma2(H, H, mul2(P2, neg1));
        float px, py, qx, qy;
        unpack2(P2, px, py);
        unpack2(Q2, qx, qy);
        float pz = hz * hz;
        float qz = fmaf(hz, hz, -pz);
        float qr = fmaf(r, r, -r2);
        float s1, e1, s2, e2, s3, e3;
        two_sum(px, py, s1, e1);
        two_sum(s1, pz, s2, e2);
        two_sum(s2, -r2, s3, e3);
        float lo = (e1 + e2) + e3;
        lo = lo + ((qx + qy) + qz);
        lo = lo - qr;
        float he = fmaf(hx, ex, fmaf(hy, ey, hz * ez));
        lo = fmaf(2.0f, he, lo);
        c = s3 + lo;
        hb = hb + fmaf(ex, R.d.x, fmaf(ey, R.d.y, ez * R.d.z));
        // f = (h + e) - s d as head + tail, then r^2 - |f|^2 compensated
        const float s = hb * R.inv_a;
        float mx = s * R.d.x, my = s * R.d.y, mz = s * R.d.z;
        float mex = fmaf(s, R.d.x, -mx), mey = fmaf(s, R.d.y, -my), mez = fmaf(s, R.d.z, -mz);
        float fx, fy, fz, fex, fey, fez;
        two_sum(hx, -mx, fx, fex);
        two_sum(hy, -my, fy, fey);
        two_sum(hz, -mz, fz, fez);
        float tx = (fex - mex) + ex, ty = (fey - mey) + ey, tz = (fez - mez) + ez;
        float gx = fx * fx, gy = fy * fy, gz = fz * fz;
        float gex = fmaf(fx, fx, -gx), gey = fmaf(fy, fy, -gy), gez = fmaf(fz, fz, -gz);
        float u1, v1, u2, v2, w, we;
        two_sum(gx, gy, u1, v1);
        two_sum(u1, gz, u2, v2);
        two_sum(r2, -u2, w, we);
        float dl = (we + qr) - (v1 + v2);
        dl = dl - ((gex + gey) + gez);
        dl = fmaf(-2.0f, fmaf(fx, tx, fmaf(fy, ty, fz * tz)), dl);
        discp = w + dl;
    } else {
        const float s = hb * R.inv_a;
        const float fx = fmaf(-s, R.d.x, hx);
        const float fy = fmaf(-s, R.d.y, hy);
        const float fz = fmaf(-s, R.d.z, hz);
        const float ff = fmaf(fx, fx, fmaf(fy, fy, fz * fz));
        discp = fmaf(r, r, -ff);
    }
    if (!(discp >= 0.0f)) return false;
    const float sd = sqrtf(R.a * discp);
    const float q = -(hb + copysignf(sd, hb));
    if (q == 0.0f) return false;
    const float ta = q * R.inv_a;
    const float tb = c / q;
    const float t0 = fminf(ta, tb), t1 = fmaxf(ta, tb);
    if (t0 >= tmin && t0 <= tmax) {
        tout = t0;
        return true;
    }
    if (t1 >= tmin && t1 <= tmax) {
        tout = t1;
        return true;
    }
    return false;
}

// ---------------------------------------------------------------------------
// Closest-hit traversal of the binary LBVH.
//
// Children are tested at their parent, from the parent's 64-byte record in
// the traversal layout (two 32-byte loads), leaves by their boxes as internal
// nodes are.  The nearer hit child is descended; the farther one's word and entry
// distance go on a per-thread stack whose first kShared entries live in shared
// memory (layout [entry][thread] so a warp touches 32 distinct banks) and the
// deeper ones in local memory.  (The walk of the wide tree below keeps its top
// entries in shared memory instead, as a ring.)  Ties on t go to the smaller slot,
// so the result does not depend on traversal order.
// ---------------------------------------------------------------------------
constexpr int kShared = 8;   // shared-memory entries per thread (power of two)
constexpr int kSharedShallow = 4;  // the fused kernel's choice for shallow trees (small scenes)
constexpr int kSpill = 72;   // local-memory entries beside those

struct StackSmem {
    int2* e;     // [kShared][block]: {node, entry distance}
};

// Counting builds only.  lane_steps / warp_steps: traversal steps summed over
// lanes, and over warps (one per step instruction the warp issues, with
// however many lanes are converged on it): their ratio / 32 is the SIMD
// utilisation of the traversal loop.
struct TraceCounters {
    uint32_t nodes, spheres, lane_steps, warp_steps;
};

// Adds a warp's counters to stats[1..4] (nodes, spheres, lane steps, warp
// steps); every lane of the warp calls it.
__device__ __forceinline__ void flush_counters(const TraceCounters& K, unsigned long long* stats) {
    unsigned long long a = K.nodes, b = K.spheres, c = K.lane_steps, d = K.warp_steps;
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
        c += __shfl_xor_sync(0xffffffffu, c, off);
        d += __shfl_xor_sync(0xffffffffu, d, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(stats + 1, a);
        atomicAdd(stats + 2, b);
        atomicAdd(stats + 3, c);
        atomicAdd(stats + 4, d);
    }
}

// Whether the ray surely does not hit the sphere it leaves again: it heads
// outwards (hb > 0), so both roots but c/q are negative, and c/q, which is at
// most -c / hb, lies below tmin > 0.  The refined c (sphere_test) differs from
// the plain one by at most (5 |h|^2 + r^2 + |c|) 2^-24, here 4 2^-24 of
// |h|^2 + r^2, and hb by at most 2^-24 |h| |d|, which is 2^-9 of it where the
// cosine is above 2^-15.  Anything not finite takes the test.
__device__ __forceinline__ bool left_behind(const RayPre& R, float4 s4, float tmin) {
    const float hx = R.o.x - s4.x, hy = R.o.y - s4.y, hz = R.o.z - s4.z;
    const float hb = fmaf(hx, R.d.x, fmaf(hy, R.d.y, hz * R.d.z));
    const float hh = fmaf(hx, hx, fmaf(hy, hy, hz * hz));
    const float r2 = s4.w * s4.w;
    return hb > 1e-15f && hb * hb > hh * R.a * 9.31322574615478515625e-10f &&      // 2^-30
           fmaf(hh + r2, -2.384185791015625e-07f, hh - r2) > hb * tmin * -0.99f;  // 2^-22
}

// Tested up front, with the whole warp converged: first the sphere the
// ray leaves (R.from; its origin lies within r/16 of that surface, so its
// test takes sphere_test's long refined branch, which in the walk would
// run at a different step in each lane), then the huge hoisted spheres
// (the ground) but that one.  Both are skipped during traversal, and
// their hit distances already cull boxes behind them.  The closest hit
// does not depend on the order of the tests.  (A scene of one sphere has
// it hoisted, see view_of.)  One copy of the test for all of them.
// Most rays leave their sphere behind; those test the ground while the others
// test the sphere they came from, and a warp without rays inside glass takes
// one round of the test instead of two (RTIOW 1920x1080 x 32 13.24 -> 13.04 ms,
// 256x144 x 4 240 -> 228 us).
template <typename T, class SV>
__device__ __forceinline__ void up_front(T& W, const SV& S, TraceCounters& K) {
    const int nh = (int)sv_nhoist(S);
    const int32_t from = W.R.from;
    int h = 0;
    if (from >= 0) {
        if (left_behind(W.R, __ldg(sv_sph(S) + from), W.tmin)) ++K.spheres;
        else h = -1;
    }
#pragma unroll 1
    for (; h < nh; ++h) {
        const int32_t k = h < 0 ? from : sv_hoist(S, h);
        if (h >= 0 && k == from) continue;
        ++K.spheres;
        W.leaf(k, __ldg(sv_sph(S) + k));
    }
}

// ---------------------------------------------------------------------------
// Two walks over the same tree.
//
// The canonical walk (CANON) tests the boxes of the canonical nodes with the
// slab test above, and every leaf's sphere; the host walk does the same, so
// its counts can be checked exactly.  It serves the counting builds and rays
// that start far outside the scene.
//
// Every other ray takes the fast walk over the traversal records (lbvh.cu):
// a box is kept as centre c and half extent h per axis, so its entry and exit
// are fma(h, -|1/d|, tc) and fma(h, |1/d|, tc) with tc = fma(c, 1/d, -p/d)
// and need no minimum and maximum per slab.  What bounds a step is issue and
// the ALU pipe (minima, maxima, compares and selects run at half the rate of
// the FMAs), and whatever one lane of a warp needs all of them pay for; so
// the x and y slabs are packed FMAs, leaves are tested by their boxes with
// the same instructions as nodes, and a sphere itself only where its box is
// hit.  A hit leaf child is descended into or pushed like a node, so spheres
// are tested nearest first and a nearer hit culls the rest: against testing
// them at once in the node's step the 1080p RTIOW frame gains 4 %, a batch of
// small renders 9 %.
//
// Nothing is lost by it.  The records hold the boxes relative to a point G in
// the middle of the scene, and so does the ray: p = o - G.  sphere_test may
// accept a point that lies off the sphere by up to 12 2^-24 (|h| + r) (h = o - C;
// roundings of h, of h.d, of the products with d and of the root), |h| + r is at
// most |p| + Q with Q the distance from G of the farthest corner of the sphere's
// box or of any box around it, and the slab parameters above are off by at most
// 2^-24 (4 Q + 6 |p|) |1/d| (1/d an ulp off, p and p/d rounded): together
// 2^-24 (16 Q + 18 |p|) in units of length.  The half extents are widened by
// 24 2^-24 (Q + E), E twice the radius around G of nearly all spheres (k_frame),
// which covers origins with |p| <= E.  For origins further out the
// rest, at most 36 2^-24 (|p| - E) max|1/d| over entry and exit, is added to the
// exit parameter as 64 2^-24 (m); where that exceeds kFarMarginMax the ray takes
// the canonical walk with margins per axis.  So neither a scene's offset nor a
// few spheres far from the others widen boxes by more than the rounding there
// asks for: with one widening for all, 1.5 2^-19 of the largest |C| + r, RTIOW
// moved by 1e6 took 67 box and 58 sphere tests a segment instead of 16 and 2.
// A box that is not finite is always met.
// ---------------------------------------------------------------------------
constexpr float kFarMarginMax = 1.0f;

// w: -2^-18 E
__device__ __forceinline__ float far_margin(f3 p, f3 inv, float w) {
    const float out = fmaxf(fmaf(fabsf(p.x) + fabsf(p.y) + fabsf(p.z), 3.814697265625e-06f, w), 0.0f);  // 2^-18
    return out * fmax3(fabsf(inv.x), fabsf(inv.y), fabsf(inv.z));
}

// The root's record behind the n - 1 node records: {c.x, c.y, h.x, h.y},
// {c.z, h.z, 0, 0}, {G, -2^-18 E}.
template <class SV>
__device__ __forceinline__ const float4* root_record(const SV& S) {
    return S.trav + 4 * (size_t)(sv_n(S) - 1u);
}

// A ray for the records of S.  G and E are read first, so that they are there
// when the reciprocals are.
template <class SV>
__device__ __forceinline__ RayPre prep_frame(const SV& S, f3 o, f3 d) {
    const bool tree = sv_n(S) > 1u;
    const float4 F = tree ? __ldg(root_record(S) + 2) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    RayPre R = prep<true>(o, d);
    // -p, x and y packed
    const f2 p_xy = fma2(pack2(R.o.x, R.o.y), pack2(-1.0f, -1.0f), pack2(F.x, F.y));
    f3 p;
    unpack2(p_xy, p.x, p.y);
    p.z = F.z - R.o.z;
    unpack2(mul2(p_xy, pack2(R.inv.x, R.inv.y)), R.n0.x, R.n0.y);
    R.n0.z = p.z * R.inv.z;
    R.m = tree ? far_margin(p, R.inv, F.w) : 0.0f;
    return R;
}

// Per-lane traversal state.  begin() prepares a ray and tests the root;
// step() tests both children of the current node (from its 64-byte record)
// and descends or pops; both return whether more work remains.  The same
// state machine serves the one-ray-per-thread kernels (trace_closest) and
// the persistent kernels that refill idle lanes.
// AXIS (canonical walk only): R carries per-axis margins.
template <bool COUNT, bool CANON = COUNT, bool AXIS = false, int KS = kShared>
struct Tracer {
    RayPre R;
    float tmin, tmax, best_t, m;
    f2 inv_xy, n0_xy, a_xy, na_xy;  // 1/d, -o/d, |1/d|, -|1/d| of x and y
    int32_t best, cur;
    int sp;
    uint32_t guard;

    __device__ __forceinline__ void leaf(int32_t k, float4 s4) {
        float t;
        if (sphere_test(R, s4, tmin, tmax, t) && (t < best_t || (t == best_t && k < best))) {
            best_t = t;
            best = k;
        }
    }

    // Entry (clipped to tmin) and exit (margin included) of a record's box.
    __device__ __forceinline__ void interval(f2 c_xy, f2 h_xy, float c_z, float h_z, float& tn, float& tf) const {
        const f2 tc = fma2(c_xy, inv_xy, n0_xy);
        float nx, ny, fx, fy;
        unpack2(fma2(h_xy, na_xy, tc), nx, ny);
        unpack2(fma2(h_xy, a_xy, tc), fx, fy);
        const float tcz = fmaf(c_z, R.inv.z, R.n0.z);
        const float nz = fmaf(h_z, -fabsf(R.inv.z), tcz), fz = fmaf(h_z, fabsf(R.inv.z), tcz);
        tn = fmaxf(fmax3(nx, ny, nz), tmin);
        tf = fmin3(fx, fy, fz);
    }
    __device__ __forceinline__ bool meets(float tn, float tf) const { return tn <= fminf(tf, best_t) + m; }

    // R_ from prep(), for the fast walk from prep_frame(); AXIS: with per-axis
    // margins.
    template <class SV>
    __device__ __forceinline__ bool begin(const SV& S, const RayPre& R_, float m_, float tmin_, float tmax_,
                                          TraceCounters& K) {
        open(R_, m_, tmin_, tmax_, tmax_, kNone);
        if (sv_n(S) == 0) return false;
        up_front(*this, S, K);
        return enter(S, K);
    }

    // A ray with the closest hit it has so far.
    __device__ __forceinline__ void open(const RayPre& R_, float m_, float tmin_, float tmax_, float t_, int32_t k_) {
        R = R_;
        m = m_;
        tmin = tmin_;
        tmax = tmax_;
        best_t = t_;
        best = k_;
        sp = 0;
    }

    // Tests the root; false: no node to walk.
    template <class SV>
    __device__ __forceinline__ bool enter(const SV& S, TraceCounters& K) {
        const uint32_t n = sv_n(S);
        if (n <= 1) return false;
        float tn;
        if (CANON) {
            float4 rlo = __ldg(sv_nodes(S) + 0), rhi = __ldg(sv_nodes(S) + 1);
            if (COUNT) ++K.nodes;
            if (!box_test<AXIS>(R, rlo, rhi, tmin, best_t, tn)) return false;
        } else {
            inv_xy = pack2(R.inv.x, R.inv.y);
            n0_xy = pack2(R.n0.x, R.n0.y);
            a_xy = pack2(fabsf(R.inv.x), fabsf(R.inv.y));
            na_xy = pack2(-fabsf(R.inv.x), -fabsf(R.inv.y));
            const float4 r0 = __ldg(root_record(S)), r1 = __ldg(root_record(S) + 1);
            float tf;
            interval(pack2(r0.x, r0.y), pack2(r0.z, r0.w), r1.x, r1.y, tn, tf);
            if (!meets(tn, tf)) return false;
        }
        cur = 0;
        // A tree has n-1 internal nodes and each step expands a different one;
        // the guard turns a cyclic (corrupt) tree into an error flag instead
        // of a hang.
        guard = 2u * n + 8u;
        return true;
    }

    // spill: this thread's local-memory stack entries beyond the KS in shared
    // memory.
    template <class SV>
    __device__ __forceinline__ bool step(const SV& S, StackSmem sm, uint32_t tid, uint32_t bdim,
                                         int2* spill, bool& overflow, TraceCounters& K) {
        // Every word of the traversal records is in range (checked when the
        // records are written), so only termination needs guarding here.
        if (--guard == 0u) {
            overflow = true;
            return false;
        }
        if (COUNT) {
            ++K.lane_steps;
            const uint32_t am = __activemask();
            if ((tid & 31u) == (uint32_t)(__ffs(am) - 1)) ++K.warp_steps;
        }
        f2 c0, h0_, z0, q0, c1, h1_, z1, q1;
        const float4* T = S.trav + 4 * (size_t)cur;
        ldg32(T, c0, h0_, z0, q0);
        ldg32(T + 2, c1, h1_, z1, q1);
        const int32_t w0 = (int32_t)(uint32_t)q0, w1 = (int32_t)(uint32_t)q1;
        bool h0 = false, h1 = false;
        float tn0 = 0.0f, tn1 = 0.0f;
        if (CANON) {
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                const int32_t w = c ? w1 : w0;
                bool h = false;
                float tn = 0.0f;
                if (w < 0) {
                    const int32_t k = w & kSlotMask;
                    if (!(w & kHoisted) && k != R.from) {
                        if (COUNT) ++K.spheres;
                        leaf(k, __ldg(sv_sph(S) + k));
                    }
                } else {
                    if (COUNT) ++K.nodes;
                    h = box_test<AXIS>(R, __ldg(sv_nodes(S) + 2 * (size_t)w), __ldg(sv_nodes(S) + 2 * (size_t)w + 1), tmin,
                                       best_t, tn);
                }
                if (c) {
                    h1 = h;
                    tn1 = tn;
                } else {
                    h0 = h;
                    tn0 = tn;
                }
            }
        } else {
            float tf0, tf1, cz, hz;
            unpack2(z0, cz, hz);
            interval(c0, h0_, cz, hz, tn0, tf0);
            unpack2(z1, cz, hz);
            interval(c1, h1_, cz, hz, tn1, tf1);
            h0 = meets(tn0, tf0);
            h1 = meets(tn1, tf1);
        }
        bool have = h0 || h1;  // cur is the next node (or, in the fast walk, leaf)
        if (have) {
            const bool second = h1 && (!h0 || tn1 < tn0);
            cur = second ? w1 : w0;
            if (h0 && h1) {
                int2 e = make_int2(second ? w0 : w1, __float_as_int(second ? tn0 : tn1));
                if (sp < KS) {
                    sm.e[(uint32_t)sp * bdim + tid] = e;
                } else {
                    if (!CANON && e.x < 0) {
                        // a far leaf goes on the stack's shared part only; beyond
                        // that it is tested first, so leaves take no entry from
                        // the nodes of deep trees
                        e = make_int2(cur, __float_as_int(second ? tn1 : tn0));
                        cur = second ? w0 : w1;
                    }
                    if (sp >= KS + kSpill) {
                        overflow = true;
                        return false;
                    }
                    spill[sp - KS] = e;
                }
                ++sp;
            }
        }
        if (!have && !pop(sm, tid, bdim, spill)) return false;
        while (!CANON && cur < 0) {
            const int32_t k = cur & kSlotMask;
            if (k != R.from) leaf(k, __ldg(sv_sph(S) + k));
            if (!pop(sm, tid, bdim, spill)) return false;
        }
        return true;
    }

    // The next entry that the closest hit so far does not cull; false: none.
    __device__ __forceinline__ bool pop(StackSmem sm, uint32_t tid, uint32_t bdim, const int2* spill) {
        while (sp > 0) {
            --sp;
            int2 e;
            if (sp < KS) e = sm.e[(uint32_t)sp * bdim + tid];
            else e = spill[sp - KS];
            if (__int_as_float(e.y) <= (CANON ? best_t : best_t + m)) {
                cur = e.x;
                return true;
            }
        }
        return false;
    }

    __device__ __forceinline__ int32_t result(float& t) const {
        if (best == kNone) {
            t = tmax;
            return -1;
        }
        t = best_t;
        return best;
    }
};

// ---------------------------------------------------------------------------
// Closest-hit traversal of the wide tree (node layout in lbvh.cu).
//
// A step loads one node and tests all of its child boxes with the same
// instructions in every lane (the fast walk's boxes and margins, with the same
// bounds: three FMAs a slab and no minimum or maximum, which run at half
// rate), pushes the hit internal children but the nearest farthest first
// onto the same shared-memory / local-memory stack as the binary traversal
// (ordered by a sorting network on keys of entry distance and child number
// when more than two are hit), tests the spheres of the leaf children whose
// boxes were hit, then descends to the nearest child unless a sphere hit now
// culls it, else pops (popped entries are culled against the closest hit).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cswap(uint32_t& a, uint32_t& b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}

// Batcher's odd-even merge sort of 4 keys, ascending.
__device__ __forceinline__ void sort4(uint32_t k[4]) {
    cswap(k[0], k[1]); cswap(k[2], k[3]);
    cswap(k[0], k[2]); cswap(k[1], k[3]);
    cswap(k[1], k[2]);
}

template <bool COUNT, int KS = kShared>
struct WideTracer {
    RayPre R;
    float tmin, tmax, best_t, m;
    int32_t best, cur;
    int sp;
    uint32_t guard;

    __device__ __forceinline__ void leaf(int32_t k, float4 s4) {
        float t;
        if (sphere_test(R, s4, tmin, tmax, t) && (t < best_t || (t == best_t && k < best))) {
            best_t = t;
            best = k;
        }
    }

    // Entry (clipped to tmin) and exit of a box.
    __device__ __forceinline__ void interval(float cx, float hx, float cy, float hy, float cz, float hz, float& tn,
                                             float& tf) const {
        const float tx = fmaf(cx, R.inv.x, R.n0.x), ty = fmaf(cy, R.inv.y, R.n0.y), tz = fmaf(cz, R.inv.z, R.n0.z);
        const float ax = fabsf(R.inv.x), ay = fabsf(R.inv.y), az = fabsf(R.inv.z);
        tn = fmaxf(fmax3(fmaf(hx, -ax, tx), fmaf(hy, -ay, ty), fmaf(hz, -az, tz)), tmin);
        tf = fmin3(fmaf(hx, ax, tx), fmaf(hy, ay, ty), fmaf(hz, az, tz));
    }
    __device__ __forceinline__ bool meets(float tn, float tf) const { return tn <= fminf(tf, best_t) + m; }

    __device__ __forceinline__ bool begin(const SceneView& S, const RayPre& R_, float m_, float tmin_, float tmax_,
                                          TraceCounters& K) {
        R = R_;
        m = m_;
        tmin = tmin_;
        tmax = tmax_;
        best_t = tmax_;
        best = kNone;
        sp = 0;
        const uint32_t n = S.n;
        if (n == 0) return false;
        up_front(*this, S, K);
        if (n == 1) return false;
        const float4 r0 = __ldg(root_record(S)), r1 = __ldg(root_record(S) + 1);
        float tn, tf;
        interval(r0.x, r0.z, r0.y, r0.w, r1.x, r1.y, tn, tf);
        if (COUNT) ++K.nodes;
        if (!meets(tn, tf)) return false;
        cur = 0;
        // every wide node is expanded at most once per ray, and there are
        // fewer than n of them: the guard turns a cyclic tree into an error
        guard = n + 8u;
        return true;
    }

    __device__ __forceinline__ void push(StackSmem sm, uint32_t tid, uint32_t bdim, int2* spill, bool& overflow,
                                         int32_t node, float tn) {
        int2* const e = sm.e + ((uint32_t)(sp & (KS - 1)) * bdim + tid);
        if (sp >= KS) {
            const int g = sp - KS;
            if (g >= kSpill) {
                overflow = true;
                return;
            }
            spill[g] = *e;
        }
        *e = make_int2(node, __float_as_int(tn));
        ++sp;
    }

    __device__ __forceinline__ bool step(const SceneView& S, StackSmem sm, uint32_t tid, uint32_t bdim,
                                         int2* spill, bool& overflow, TraceCounters& K) {
        if (--guard == 0u) {
            overflow = true;
            return false;
        }
        if (COUNT) {
            ++K.lane_steps;
            const uint32_t am = __activemask();
            if ((tid & 31u) == (uint32_t)(__ffs(am) - 1)) ++K.warp_steps;
        }
        const float4* N = S.wide + kWideF4 * (size_t)cur;
        // key of child c: its entry distance's bits with c in the low three
        // bits (distances are >= tmin > 0, so the bits order like the
        // values; the cut makes a key's distance a lower bound), all ones
        // unless it is a hit internal child.  Unused entries and hoisted
        // leaves have empty boxes.
        uint32_t key[kWideW];
        uint32_t lhit = 0;
        const int32_t* words = reinterpret_cast<const int32_t*>(N + 6);
        {
            const int4 w4 = __ldg(reinterpret_cast<const int4*>(words));
            if (COUNT) K.nodes += (w4.x >= 0) + (w4.y >= 0) + (w4.z >= 0) + (w4.w >= 0);
            f2 cx01, cx23, hx01, hx23, cy01, cy23, hy01, hy23, cz01, cz23, hz01, hz23;
            ldg32(N, cx01, cx23, hx01, hx23);
            ldg32(N + 2, cy01, cy23, hy01, hy23);
            ldg32(N + 4, cz01, cz23, hz01, hz23);
#define VENU_WIDE_PAIR(P, I, W0, W1)                                                                  \
    {                                                                                                 \
        float cxa, cxb, hxa, hxb, cya, cyb, hya, hyb, cza, czb, hza, hzb, tn, tf;                     \
        unpack2(cx##P, cxa, cxb);                                                                     \
        unpack2(hx##P, hxa, hxb);                                                                     \
        unpack2(cy##P, cya, cyb);                                                                     \
        unpack2(hy##P, hya, hyb);                                                                     \
        unpack2(cz##P, cza, czb);                                                                     \
        unpack2(hz##P, hza, hzb);                                                                     \
        interval(cxa, hxa, cya, hya, cza, hza, tn, tf);                                               \
        bool ok = meets(tn, tf);                                                                      \
        lhit |= (uint32_t)(ok && (W0) < 0) << (I);                                                    \
        key[I] = ok && (W0) >= 0 ? (__float_as_uint(tn) & ~7u) | (uint32_t)(I) : 0xffffffffu;         \
        interval(cxb, hxb, cyb, hyb, czb, hzb, tn, tf);                                               \
        ok = meets(tn, tf);                                                                           \
        lhit |= (uint32_t)(ok && (W1) < 0) << ((I) + 1);                                              \
        key[(I) + 1] = ok && (W1) >= 0 ? (__float_as_uint(tn) & ~7u) | (uint32_t)((I) + 1) : 0xffffffffu; \
    }
            VENU_WIDE_PAIR(01, 0, w4.x, w4.y)
            VENU_WIDE_PAIR(23, 2, w4.z, w4.w)
#undef VENU_WIDE_PAIR
        }
        // the hit internal children but the nearest onto the stack, farthest
        // first (one or two hits without sorting); the nearest is descended
        // unless the leaf tests below cull it
        uint32_t kmin = key[0];
#pragma unroll
        for (int c = 1; c < kWideW; ++c) kmin = min(kmin, key[c]);
        if (kmin != 0xffffffffu) {
            uint32_t nhit = 0;
#pragma unroll
            for (int c = 0; c < kWideW; ++c) nhit += key[c] != 0xffffffffu;
            if (nhit == 2u) {
                uint32_t kmax = 0;
#pragma unroll
                for (int c = 0; c < kWideW; ++c) kmax = key[c] != 0xffffffffu ? max(kmax, key[c]) : kmax;
                push(sm, tid, bdim, spill, overflow, __ldg(words + (kmax & 7u)),
                     __uint_as_float(kmax & ~7u));
            } else if (nhit > 2u) {
                sort4(key);
#pragma unroll
                for (int i = kWideW - 1; i >= 1; --i) {
                    if (key[i] != 0xffffffffu)
                        push(sm, tid, bdim, spill, overflow, __ldg(words + (key[i] & 7u)),
                             __uint_as_float(key[i] & ~7u));
                }
            }
            if (overflow) return false;
        }
        // then the spheres of the hit leaf children, which may shorten the
        // ray and cull the pushed entries and the nearest child
        for (uint32_t lm = lhit; lm; lm &= lm - 1u) {
            const int32_t k = __ldg(words + (__ffs(lm) - 1)) & kSlotMask;
            if (k != R.from) {
                if (COUNT) ++K.spheres;
                leaf(k, __ldg(S.sph + k));
            }
        }
        if (kmin != 0xffffffffu && __uint_as_float(kmin & ~7u) <= best_t + m) {
            cur = __ldg(words + (kmin & 7u));
            return true;
        }
        while (sp > 0) {
            --sp;
            int2* const p = sm.e + ((uint32_t)(sp & (KS - 1)) * bdim + tid);
            const int2 e = *p;
            if (sp >= KS) *p = spill[sp - KS];
            if (__int_as_float(e.y) <= best_t + m) {
                cur = e.x;
                return true;
            }
        }
        return false;
    }

    __device__ __forceinline__ int32_t result(float& t) const {
        if (best == kNone) {
            t = tmax;
            return -1;
        }
        t = best_t;
        return best;
    }
};

template <bool COUNT, bool WIDE = false, class SV>
__device__ __forceinline__ RayPre prep_for(const SV& S, f3 o, f3 d) {
    if constexpr (COUNT && !WIDE) return prep<false>(o, d);
    else return prep_frame(S, o, d);
}

template <class T, class SV>
__device__ __forceinline__ int32_t trace_with(const SV& S, const RayPre& R, float m, float tmin, float tmax,
                                              float& t_out, StackSmem sm, uint32_t tid, uint32_t bdim,
                                              bool& overflow, TraceCounters& K) {
    T W;
    int2 spill[kSpill];
    if (W.begin(S, R, m, tmin, tmax, K))
        while (W.step(S, sm, tid, bdim, spill, overflow, K)) {
        }
    return W.result(t_out);
}

// Closest hit of one ray (R from prep_for<COUNT, WIDE>): the fast walk, over
// the binary or the wide tree.  Rays that start far outside the scene (rare)
// take the canonical walk with per-axis margins; counting builds of the binary
// tree the canonical walk with one margin, or per axis for the rare
// near-axis-parallel ray.  KS: shared-memory stack entries per thread (the
// kernel's StackSmem holds KS of them).
template <bool COUNT, int KS = kShared, bool WIDE = false, class SV>
__device__ __forceinline__ int32_t trace_closest(const SV& S, const RayPre& R, float tmin,
                                                 float tmax, float& t_out, StackSmem sm,
                                                 uint32_t tid, uint32_t bdim, bool& overflow,
                                                 TraceCounters& K) {
    if (COUNT && !WIDE ? R.axis : !(R.m <= kFarMarginMax)) {
        RayPre A = prep<false>(R.o, R.d);
        A.from = R.from;
        axis_margins(A);
        return trace_with<Tracer<COUNT, true, true, KS>>(S, A, 0.0f, tmin, tmax, t_out, sm, tid, bdim, overflow, K);
    }
    if constexpr (WIDE)
        return trace_with<WideTracer<COUNT, KS>>(S, R, R.m, tmin, tmax, t_out, sm, tid, bdim, overflow, K);
    return trace_with<Tracer<COUNT, COUNT, false, KS>>(S, R, R.m, tmin, tmax, t_out, sm, tid, bdim, overflow, K);
}

// ---------------------------------------------------------------------------
// Path state in the wavefront queues (48 bytes per path; 52 in the batch
// engine):
//   o4 = {origin.xyz, slot (int bits)}
//   d4 = {direction.xyz, remaining depth (bits 0-7) | job index (batch
//         engine) or 1 + slot of the sphere the ray leaves (single-scene
//         renderer) (bits 8-31)}
//   t4 = {throughput.rgb, bounce seed (uint bits)}
//   from = the batch engine's slot of the sphere the ray leaves
//          (RayPre::from), -1 for a camera ray; null in the single-scene
//          renderer
// ---------------------------------------------------------------------------
struct Queue {
    float4* o;
    float4* d;
    float4* t;
    int32_t* from;
};

}  // namespace venu
