// vgb_device.cuh -- device helpers of the hot path: counter-based RNG, the reference's FP32
// expression order, the watertight ray/triangle test and BVH traversal.
//
// The translation unit is compiled with --fmad=false: every `a * b + c` below rounds the
// product and the sum separately, exactly as the oracle (built with -ffp-contract=off) and
// the reference's glm code do.  Fused multiply-adds appear only where written explicitly.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/vgb.h"
#include "vgb_internal.h"

namespace vgbd {

constexpr float kPi = 3.14159265358979323846f;
constexpr float kInvPi = (float)(1. / 3.141592653589793238462);
constexpr uint32_t kSlotMain = 0u, kSlotRR = 0xFEu, kSlotJitter = 0xFFu;

// device error word bits
constexpr uint32_t kErrStack = 1u, kErrIter = 2u;

constexpr int kStackSize = 64;   // binary layout
constexpr uint32_t kIterCap = 1u << 22;  // default traversal steps per ray before giving up

// ------------------------------------------------------------------ Philox-4x32-10
// Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3", SC 2011.
struct U4 { uint32_t x, y, z, w; };
__device__ __forceinline__ U4 philox(U4 c, uint32_t k0, uint32_t k1) {
    const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) { k0 += W0; k1 += W1; }
        uint32_t hi0 = __umulhi(M0, c.x), lo0 = M0 * c.x;
        uint32_t hi1 = __umulhi(M1, c.z), lo1 = M1 * c.z;
        c = U4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
    }
    return c;
}
__device__ __forceinline__ float u01(uint32_t x) { return (float)(x >> 8) * (1.0f / 16777216.0f); }

// std::max / std::min semantics (first argument wins on NaN comparisons)
__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }

struct F3 { float x, y, z; };
__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator*(float s, F3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ F3 operator*(F3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float dot(F3 a, F3 b) { return (a.x * b.x + a.y * b.y) + a.z * b.z; }
__device__ __forceinline__ F3 cross(F3 a, F3 b) {
    return {a.y * b.z - b.y * a.z, a.z * b.x - b.z * a.x, a.x * b.y - b.x * a.y};
}
__device__ __forceinline__ float length(F3 a) { return sqrtf(dot(a, a)); }
__device__ __forceinline__ F3 normalize(F3 a) { return a * (1.0f / sqrtf(dot(a, a))); }
__device__ __forceinline__ float pick(F3 a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : a.z); }
__device__ __forceinline__ F3 ld3(const float4& v) { return F3{v.x, v.y, v.z}; }

// offsetIntersection, float path (include/implementation/rendering/ray.ipp:107-123)
__device__ __forceinline__ float offset1(float p, float n) {
    const float origin = 1.f / 32.f, float_scale = 1.f / 65536.f, int_scale = 256.f;
    int32_t of = (int32_t)(int_scale * n);
    int32_t pi = __float_as_int(p) + ((p < 0) ? -of : of);
    return (fabsf(p) < origin) ? p + float_scale * n : __int_as_float(pi);
}

// ------------------------------------------------------------------ watertight test
// Woop, Benthin, Wald, "Watertight Ray/Triangle Intersection", JCGT 2(1), 2013.
struct WRay {
    F3 o, d;
    int kx, ky, kz;
    float Sx, Sy, Sz;
};

__device__ __forceinline__ float safe_rcp(float d) {
    const float tiny = 1e-30f;
    float a = fabsf(d) < tiny ? copysignf(tiny, d) : d;
    return 1.0f / a;
}

__device__ __forceinline__ WRay make_wray(F3 o, F3 d) {
    WRay r;
    r.o = o; r.d = d;
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz + 1; if (kx == 3) kx = 0;
    int ky = kx + 1; if (ky == 3) ky = 0;
    if (pick(d, kz) < 0.0f) { int t = kx; kx = ky; ky = t; }
    r.kx = kx; r.ky = ky; r.kz = kz;
    float dz = pick(d, kz);
    r.Sx = pick(d, kx) / dz;
    r.Sy = pick(d, ky) / dz;
    r.Sz = 1.0f / dz;
    return r;
}

// Returns false on a miss.  t > 0 required.  U, V, W: unnormalised weights of v0, v1, v2.
__device__ __forceinline__ bool wt_test(const WRay& r, F3 v0, F3 v1, F3 v2, float& t_out, float& U_out,
                                        float& V_out, float& W_out, float& det_out) {
    F3 A = v0 - r.o, B = v1 - r.o, C = v2 - r.o;
    float Akz = pick(A, r.kz), Bkz = pick(B, r.kz), Ckz = pick(C, r.kz);
    float Ax = pick(A, r.kx) - r.Sx * Akz;
    float Ay = pick(A, r.ky) - r.Sy * Akz;
    float Bx = pick(B, r.kx) - r.Sx * Bkz;
    float By = pick(B, r.ky) - r.Sy * Bkz;
    float Cx = pick(C, r.kx) - r.Sx * Ckz;
    float Cy = pick(C, r.ky) - r.Sy * Ckz;
    float U = Cx * By - Cy * Bx;
    float V = Ax * Cy - Ay * Cx;
    float W = Bx * Ay - By * Ax;
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        double CxBy = (double)Cx * (double)By, CyBx = (double)Cy * (double)Bx;
        U = (float)(CxBy - CyBx);
        double AxCy = (double)Ax * (double)Cy, AyCx = (double)Ay * (double)Cx;
        V = (float)(AxCy - AyCx);
        double BxAy = (double)Bx * (double)Ay, ByAx = (double)By * (double)Ax;
        W = (float)(BxAy - ByAx);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    float det = U + V + W;
    if (det == 0.0f) return false;
    float T = (U * (r.Sz * Akz) + V * (r.Sz * Bkz)) + W * (r.Sz * Ckz);
    float t = T * (1.0f / det);
    if (!(t > 0.0f)) return false;
    t_out = t; U_out = U; V_out = V; W_out = W; det_out = det;
    return true;
}

// ------------------------------------------------------------------ BVH2 traversal
struct HitOut {
    float t;
    uint32_t id;
    float U, V, W, det;
};

struct Counters { uint32_t nodes, tris; };

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float fmin3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Per-ray constants of the slab test.  A plane distance is one fused multiply-add,
// fma(plane, 1/d, -(o/d) -+ e): with o/d rounded once, its error is a relative part below
// 2^-23 (the reciprocal and the fma) plus an absolute part below 2^-24 |o/d|, so each axis
// shifts its near plane down and its far plane up by e = 2^-20 |o/d| (16x that bound), and the
// exit distance is widened by 2^-20 for the relative part (Ize 2013).  No box that the exact
// slab test keeps is culled, so the closest hit does not depend on this arithmetic.
struct SlabRay {
    float ix, iy, iz, lx, hx, ly, hy, lz, hz;  // reciprocals; offsets of the lo and hi planes
};
__device__ __forceinline__ SlabRay make_slab(const WRay& r) {
    SlabRay q;
    q.ix = safe_rcp(r.d.x); q.iy = safe_rcp(r.d.y); q.iz = safe_rcp(r.d.z);
    const float ox = r.o.x * q.ix, oy = r.o.y * q.iy, oz = r.o.z * q.iz;
    const float ex = fabsf(ox) * 0x1p-20f, ey = fabsf(oy) * 0x1p-20f, ez = fabsf(oz) * 0x1p-20f;
    q.lx = (q.ix >= 0.f) ? (-ox - ex) : (-ox + ex);
    q.hx = (q.ix >= 0.f) ? (-ox + ex) : (-ox - ex);
    q.ly = (q.iy >= 0.f) ? (-oy - ey) : (-oy + ey);
    q.hy = (q.iy >= 0.f) ? (-oy + ey) : (-oy - ey);
    q.lz = (q.iz >= 0.f) ? (-oz - ez) : (-oz + ez);
    q.hz = (q.iz >= 0.f) ? (-oz + ez) : (-oz - ez);
    return q;
}

// Entry and exit distances of the box [lo, hi] clipped to [0, tfar] (exit widened).
__device__ __forceinline__ void slab(const SlabRay& q, float lox, float hix, float loy, float hiy, float loz,
                                     float hiz, float tfar, float& tn, float& tf) {
    const float widen = 1.0f + 0x1p-20f;
    const float a0 = fmaf(lox, q.ix, q.lx), a1 = fmaf(hix, q.ix, q.hx);
    const float b0 = fmaf(loy, q.iy, q.ly), b1 = fmaf(hiy, q.iy, q.hy);
    const float c0 = fmaf(loz, q.iz, q.lz), c1 = fmaf(hiz, q.iz, q.hz);
    tn = fmax3(fminf(a0, a1), fminf(b0, b1), fmaxf(fminf(c0, c1), 0.0f));
    tf = fmin3(fmaxf(a0, a1), fmaxf(b0, b1), fminf(fmaxf(c0, c1), tfar)) * widen;
}

// Occlusion on the binary nodes: the first triangle met with t <= tmax.  vgb_trace_rays reports that
// triangle, so its walk keeps this tree's order; every other ray walks the wide nodes below.  Box tests
// are conservative (make_slab).
template <bool COUNT>
__device__ __forceinline__ void occluded2(const float4* __restrict__ nodes, const float4* __restrict__ tris,
                                          const WRay& r, float tmax, HitOut& h, uint32_t& err, Counters& cnt,
                                          uint32_t cap) {
    int stack[kStackSize];
    int sp = 0;
    int node = 0;
    h.t = __int_as_float(0x7f800000);
    h.id = VGB_NO_HIT;
    uint32_t iter = 0;
    const SlabRay q = make_slab(r);
    while (true) {
        while (node >= 0) {
            if (++iter > cap) { err |= kErrIter; return; }
            const float4 n0 = __ldg(&nodes[4 * node + 0]);
            const float4 n1 = __ldg(&nodes[4 * node + 1]);
            const float4 n2 = __ldg(&nodes[4 * node + 2]);
            const float4 n3 = __ldg(&nodes[4 * node + 3]);
            if (COUNT) cnt.nodes++;
            float tn0, tf0, tn1, tf1;
            slab(q, n0.x, n0.y, n0.z, n0.w, n2.x, n2.y, tmax, tn0, tf0);
            slab(q, n1.x, n1.y, n1.z, n1.w, n2.z, n2.w, tmax, tn1, tf1);
            const bool h0 = tn0 <= tf0, h1 = tn1 <= tf1;
            const int ch0 = __float_as_int(n3.x), ch1 = __float_as_int(n3.y);
            if (h0 && h1) {
                int nearc = ch0, farc = ch1;
                if (tn1 < tn0) { nearc = ch1; farc = ch0; }
                if (sp >= kStackSize) { err |= kErrStack; return; }
                stack[sp++] = farc;
                node = nearc;
            } else if (h0) {
                node = ch0;
            } else if (h1) {
                node = ch1;
            } else {
                if (sp == 0) return;
                node = stack[--sp];
            }
        }
        // leaf
        const uint32_t x = ~(uint32_t)node;
        const uint32_t start = x >> 3, cntl = (x & 7u) + 1u;
        for (uint32_t k = 0; k < cntl; ++k) {
            const float4 t0 = __ldg(&tris[3 * (start + k) + 0]);
            const float4 t1 = __ldg(&tris[3 * (start + k) + 1]);
            const float4 t2 = __ldg(&tris[3 * (start + k) + 2]);
            if (COUNT) cnt.tris++;
            float tt, U, V, W, det;
            if (wt_test(r, ld3(t0), ld3(t1), ld3(t2), tt, U, V, W, det) && tt <= tmax) {
                h.t = tt;
                h.id = __float_as_uint(t0.w);
                return;
            }
        }
        if (sp == 0) return;
        node = stack[--sp];
    }
}

// ------------------------------------------------------------------ wide traversal (4 children per node)
// The layout the render, batch, adjoint and closest-hit ray kernels walk: the binary tree with
// up to three inner nodes folded into one 128-byte node (one cache line; WideNode in
// vgb_internal.h), so a ray follows half as many dependent node fetches.  A child's box is its
// centre c and half extent h: with m = (c - o) / d, the entry and exit of an axis are m - h / |d|
// and m + h / |d|, which needs no per-axis minimum and maximum, and the four operations run two
// lanes wide (f32x2).  The binary traversal was bound by the latency of its chain of node fetches
// and by the ALU pipe that executes minimum, maximum and select (47 % busy against 17 % of the
// FMA pipe at camera rays).
// Nodes visited per ray 24.3 -> 12.3 (8.4M triangles, camera and bounce rays);
// whole calls: 512^2 x 16 spp over 2.1M triangles 7.96 -> 7.32 ms, 2048^2 x 4 spp over 8.4M 14.1 ->
// 13.5 ms, fused adjoint of 12 asteroid views 9.0 -> 7.8 ms.  Folding three nodes beat the same
// box test on the binary nodes (7.91 against 7.38 ms of device time at 512^2, 13.38 against 13.15
// at 2048^2); walking the children of occlusion rays unsorted lost (2.94 -> 3.16 ms at 512^2).
//
// Conservative: m carries a relative error below 6 * 2^-24, so a plane distance m -+ h / |d| is
// off by at most that part of |distance| + h / |d|; the builder enlarges h (wide_half_extent) by
// far more than the second part, and the exit distance is widened by 2^-18 for the first, which
// also covers the rounding of the triangle test's own distance and edge functions.  No box that
// holds a triangle the test accepts is culled, so the closest hit does not depend on the layout.
using vgb::kStackWide;
constexpr int kWideEmpty = (int)0x80000000; // link of an empty child slot; the stack's bottom entry

typedef unsigned long long u64;
__device__ __forceinline__ u64 pk2(float lo, float hi) {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void up2(u64 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// 32 bytes (a 32-byte aligned address) in one load.
__device__ __forceinline__ void ldg32(const void* p, u64& a, u64& b, u64& c, u64& d) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// The box test runs in distances scaled by kWideTime (a power of two: nothing is rounded by it).  A
// direction component of 0 counts as 1e-30, and in unscaled distances (c - o) / d then overflows from
// |c - o| = 3.4e8 on: with the centre at -infinity the exit is there too, and a box that holds the ray
// would be culled.  Scaled, that takes 6e27, beyond what the triangle test's products hold, and a
// distance only turns subnormal below 2e-19, far under the boxes' margins.  A direction of any length
// (UNIT false) is divided by its largest component first, |1 / Sz| of the triangle test; the rounding of
// that is part of the margins below.
constexpr float kWideTime = 0x1p-64f;
template <bool UNIT>
__device__ __forceinline__ float wide_time(const WRay& r, float t) {
    return UNIT ? t * kWideTime : t / fabsf(r.Sz) * kWideTime;
}

// kWideTime / |d| to one unit in the last place, d clamped away from 0: enough for the box test's margins.
__device__ __forceinline__ float wide_rcp(float d) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fabsf(d)));
    return fminf(r * kWideTime, 1e30f * kWideTime);
}

// Per-ray constants: minus the origin, 1/d and +-1/|d|, the x and y axes as a pair, z twice.
struct WideRay { u64 noxy, nozz, ixy, izz, axy, azz, nxy, nzz; };
template <bool UNIT = true>
__device__ __forceinline__ WideRay make_wide(const WRay& r) {
    WideRay q;
    const F3 d = UNIT ? r.d : r.d * fabsf(r.Sz);
    const float ix = copysignf(wide_rcp(d.x), d.x), iy = copysignf(wide_rcp(d.y), d.y), iz = copysignf(wide_rcp(d.z), d.z);
    const float ax = fabsf(ix), ay = fabsf(iy), az = fabsf(iz);
    q.noxy = pk2(-r.o.x, -r.o.y); q.nozz = pk2(-r.o.z, -r.o.z);
    q.ixy = pk2(ix, iy); q.izz = pk2(iz, iz);
    q.axy = pk2(ax, ay); q.azz = pk2(az, az);
    q.nxy = pk2(-ax, -ay); q.nzz = pk2(-az, -az);
    return q;
}

// State of one ray's traversal between calls (the stack lives in the caller's per-thread array).
struct TravState {
    int node;       // next node (>= 0 inner; < 0 a leaf to test; kWideEmpty: finished)
    int sp;         // stack entries, the bottom one included
    float best;     // closest-hit t so far (tmax for occlusion rays), in the box test's distances
    uint32_t iter;  // nodes visited
};

template <bool UNIT = true>
__device__ __forceinline__ TravState trav_start(const WRay& r, float tmax, bool any, HitOut& h, int* stack) {
    h.t = __int_as_float(0x7f800000);
    h.id = VGB_NO_HIT;
    stack[0] = kWideEmpty;
    return TravState{0, 1, any ? wide_time<UNIT>(r, tmax) : __int_as_float(0x7f800000), 0u};
}

// Closest hit (any = false; ties in t go to the smaller id) or occlusion (any = true, any hit
// with t <= tmax).  The stack holds any walk of a tree that the build accepts (kWideLevels levels, three
// pushes each), so pushes need no test; a ray over its step cap is stopped where it next takes a node
// off the stack, which bounds it as well: a descent between two of those is as long as the tree is deep.
// (Testing both at every node cost 1-2 %: 512^2 x 16 spp 2.36 against 2.32 ms.)  RESUME: stops after
// `budget` nodes; returns true when the ray is finished (h holds its answer), false when the next call is to
// continue from ts.
template <bool COUNT, bool RESUME, bool UNIT = true>
__device__ __forceinline__ bool traverse4(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                          const WRay& r, const WideRay& q, float tmax, const bool any, int* stack,
                                          TravState& ts, HitOut& h, uint32_t& err, Counters& cnt, uint32_t cap,
                                          int budget) {
    const u64 widen = pk2(1.0f + 0x1p-18f, 1.0f + 0x1p-18f);
    const float inf = __int_as_float(0x7f800000);
    int node = ts.node, sp = ts.sp;
    float best = ts.best;
    uint32_t iter = ts.iter;
    while (true) {
        while (node >= 0) {
            if (RESUME && budget-- <= 0) {
                ts.node = node; ts.sp = sp; ts.best = best; ts.iter = iter;
                return false;
            }
            ++iter;
            const char* p = reinterpret_cast<const char*>(nodes) + (size_t)(uint32_t)node * 128u;
            u64 c0, h0, c1, h1, c2, h2, c3, h3, cz01, cz23, hz01, hz23;
            ldg32(p, c0, h0, c1, h1);
            ldg32(p + 32, c2, h2, c3, h3);
            ldg32(p + 64, cz01, cz23, hz01, hz23);
            const int4 link = __ldg(reinterpret_cast<const int4*>(p + 96));
            if (COUNT) cnt.nodes++;
            float tn[4], tf[4];
            {
                const u64 m01 = mul2(add2(cz01, q.nozz), q.izz), m23 = mul2(add2(cz23, q.nozz), q.izz);
                up2(fma2(hz01, q.nzz, m01), tn[0], tn[1]);
                up2(fma2(hz23, q.nzz, m23), tn[2], tn[3]);
                up2(fma2(hz01, q.azz, m01), tf[0], tf[1]);
                up2(fma2(hz23, q.azz, m23), tf[2], tf[3]);
            }
            const u64 cc[4] = {c0, c1, c2, c3}, hh[4] = {h0, h1, h2, h3};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const u64 m = mul2(add2(cc[k], q.noxy), q.ixy);
                float nx, ny, fx, fy;
                up2(fma2(hh[k], q.nxy, m), nx, ny);
                up2(fma2(hh[k], q.axy, m), fx, fy);
                tn[k] = fmax3(nx, ny, fmaxf(tn[k], 0.0f));
                tf[k] = fmin3(fx, fy, fminf(tf[k], best));
            }
            up2(mul2(pk2(tf[0], tf[1]), widen), tf[0], tf[1]);
            up2(mul2(pk2(tf[2], tf[3]), widen), tf[2], tf[3]);
            const bool b0 = tn[0] <= tf[0], b1 = tn[1] <= tf[1], b2 = tn[2] <= tf[2], b3 = tn[3] <= tf[3];
            const int l0 = b0 ? link.x : kWideEmpty, l1 = b1 ? link.y : kWideEmpty;
            const int l2 = b2 ? link.z : kWideEmpty, l3 = b3 ? link.w : kWideEmpty;
            // near to far: each pair by its entry distances, then the pairs by their nearer one
            const float t0 = b0 ? tn[0] : inf, t1 = b1 ? tn[1] : inf, t2 = b2 ? tn[2] : inf, t3 = b3 ? tn[3] : inf;
            const bool s01 = t1 < t0, s23 = t3 < t2;
            const int a0 = s01 ? l1 : l0, a1 = s01 ? l0 : l1, e0 = s23 ? l3 : l2, e1 = s23 ? l2 : l3;
            const bool sw = fminf(t2, t3) < fminf(t0, t1);
            const int n0 = sw ? e0 : a0, n1 = sw ? e1 : a1, f0 = sw ? a0 : e0, f1 = sw ? a1 : e1;
            if (f1 != kWideEmpty) stack[sp++] = f1;
            if (f0 != kWideEmpty) stack[sp++] = f0;
            if (n1 != kWideEmpty) stack[sp++] = n1;
            node = n0;
            if (node == kWideEmpty) {
                if (iter > cap) { err |= kErrIter; return true; }
                node = stack[--sp];
            }
        }
        if (node == kWideEmpty) {
            if (iter > cap) err |= kErrIter;
            return true;
        }
        const uint32_t x = ~(uint32_t)node;
        const uint32_t start = x >> 3, cntl = (x & 7u) + 1u;
        for (uint32_t k = 0; k < cntl; ++k) {
            const float4 t0 = __ldg(&tris[3 * (start + k) + 0]);
            const float4 t1 = __ldg(&tris[3 * (start + k) + 1]);
            const float4 t2 = __ldg(&tris[3 * (start + k) + 2]);
            if (COUNT) cnt.tris++;
            float tt, U, V, W, det;
            if (wt_test(r, ld3(t0), ld3(t1), ld3(t2), tt, U, V, W, det)) {
                const uint32_t id = __float_as_uint(t0.w);
                if (any) {
                    if (tt <= tmax) {
                        h.t = tt; h.id = id;
                        if (iter > cap) err |= kErrIter;
                        return true;
                    }
                } else if (tt < h.t || (tt == h.t && id < h.id)) {
                    h.t = tt; h.id = id; h.U = U; h.V = V; h.W = W; h.det = det;
                    best = wide_time<UNIT>(r, tt);
                }
            }
        }
        node = stack[--sp];
    }
}

template <bool COUNT, bool UNIT = true>
__device__ __forceinline__ void traverse4_rt(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                             const WRay& r, float tmax, const bool any, HitOut& h, uint32_t& err,
                                             Counters& cnt, uint32_t cap) {
    int stack[kStackWide];
    TravState ts = trav_start<UNIT>(r, tmax, any, h, stack);
    traverse4<COUNT, false, UNIT>(nodes, tris, r, make_wide<UNIT>(r), tmax, any, stack, ts, h, err, cnt, cap, 0);
}

// ------------------------------------------------------------------ compressed 8-wide traversal
// Node (80 bytes, five 16-byte words): origin p, biased exponents and internal-child mask,
// first internal child, first triangle, eight meta bytes and six arrays of eight 8-bit
// quantised bounds.  The child in slot s is the nearest for rays whose direction-sign octant
// is s; a ray of octant o visits slots o^0, o^1, ..., o^7.  The stack holds node groups: the
// first child index, the internal-child mask and the not-yet-visited hit slots in visiting order.
constexpr int kStack8 = 32;

__device__ __forceinline__ uint32_t octant_order(uint32_t m, uint32_t o) {
    // bit k of the result = bit (o ^ k) of m
    if (o & 1u) m = ((m & 0x55u) << 1) | ((m & 0xAAu) >> 1);
    if (o & 2u) m = ((m & 0x33u) << 2) | ((m & 0xCCu) >> 2);
    if (o & 4u) m = ((m & 0x0Fu) << 4) | ((m & 0xF0u) >> 4);
    return m;
}

// Quantised coordinate `byte` of w as a float, exactly: the byte goes into the mantissa of
// 2^23 (byte permute) and 2^23 is subtracted, so no integer-to-float conversion is issued.
__device__ __forceinline__ float q8(uint32_t w, int byte) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u | (uint32_t)byte)) - 8388608.0f;
}

// Nonzero bytes of w as a 4-bit mask (bit k: byte k != 0).
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
    const uint32_t m = ((w & 0x7F7F7F7Fu) + 0x7F7F7F7Fu | w) & 0x80808080u;
    return ((m >> 7) & 1u) | ((m >> 14) & 2u) | ((m >> 21) & 4u) | ((m >> 28) & 8u);
}

// Plane distances of one node axis for the ray: t(q) = fma(q, a, b -+ e) with a = 2^e_axis / d
// (exact) and b = (p - o) / d.  Against (p + 2^e q - o) / d in exact arithmetic the error is a
// relative part below 2^-23 (the final fma and the relative part of b), an absolute part below
// 2^-23 |b| (b's two roundings) and, because the builder bounds the FP32-rounded dequantised
// plane, not the exact one, an absolute part below 2^-24 |p + 2^e q| / |d|.  The margin
// e = 2^-20 (|b| + |1/d| (|p| + 255 * 2^e)) covers the absolute parts 8x; the relative part is
// covered by widening the exit distance by 2^-20, as in the binary test.
struct AxisPlanes { float a, bn, bf; };
__device__ __forceinline__ AxisPlanes axis_planes(float p, float s, float o, float inv) {
    const float a = s * inv;
    const float b = (p - o) * inv;
    const float e = 0x1p-20f * fmaf(fabsf(inv), fmaf(255.0f, s, fabsf(p)), fabsf(b));
    return AxisPlanes{a, b - e, b + e};
}

template <bool COUNT>
__device__ __forceinline__ void traverse8_rt(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                             const WRay& r, float tmax, const bool any, HitOut& h, uint32_t& err,
                                             Counters& cnt, uint32_t cap) {
    const float widen = 1.0f + 0x1p-20f;
    const uint32_t oct = (r.d.x < 0.f ? 1u : 0u) | (r.d.y < 0.f ? 2u : 0u) | (r.d.z < 0.f ? 4u : 0u);
    // the near plane of an axis is the box's low side for a positive reciprocal, else the high side
    const float ix = safe_rcp(r.d.x), iy = safe_rcp(r.d.y), iz = safe_rcp(r.d.z);
    const bool nx = ix < 0.f, ny = iy < 0.f, nz = iz < 0.f;
    uint2 stack[kStack8];
    int sp = 0;
    uint32_t node = 0;
    float best = any ? tmax : __int_as_float(0x7f800000);
    h.t = __int_as_float(0x7f800000);
    h.id = VGB_NO_HIT;
    uint32_t iter = 0;
    while (true) {
        if (++iter > cap) { err |= kErrIter; return; }
        const uint4 w0 = __ldg(&nodes[5 * node + 0]);
        const uint4 w1 = __ldg(&nodes[5 * node + 1]);
        const uint4 w2 = __ldg(&nodes[5 * node + 2]);
        const uint4 w3 = __ldg(&nodes[5 * node + 3]);
        const uint4 w4 = __ldg(&nodes[5 * node + 4]);
        if (COUNT) cnt.nodes++;
        const AxisPlanes X = axis_planes(__uint_as_float(w0.x), __uint_as_float((w0.w & 0xFFu) << 23), r.o.x, ix);
        const AxisPlanes Y = axis_planes(__uint_as_float(w0.y), __uint_as_float(((w0.w >> 8) & 0xFFu) << 23), r.o.y, iy);
        const AxisPlanes Z = axis_planes(__uint_as_float(w0.z), __uint_as_float(((w0.w >> 16) & 0xFFu) << 23), r.o.z, iz);
        const uint32_t imask = w0.w >> 24;
        const uint32_t child_base = w1.x, tri_base = w1.y;
        const uint32_t valid = nonzero_bytes(w1.z) | (nonzero_bytes(w1.w) << 4);
        // quantised near / far planes per axis, slots 0-3 and 4-7
        const uint32_t nx0 = nx ? w3.z : w2.x, nx1 = nx ? w3.w : w2.y, fx0 = nx ? w2.x : w3.z, fx1 = nx ? w2.y : w3.w;
        const uint32_t ny0 = ny ? w4.x : w2.z, ny1 = ny ? w4.y : w2.w, fy0 = ny ? w2.z : w4.x, fy1 = ny ? w2.w : w4.y;
        const uint32_t nz0 = nz ? w4.z : w3.x, nz1 = nz ? w4.w : w3.y, fz0 = nz ? w3.x : w4.z, fz1 = nz ? w3.y : w4.w;
        uint32_t hits = 0;
#pragma unroll
        for (int sl = 0; sl < 8; ++sl) {
            const int b = sl & 3;
            const float tnx = fmaf(q8(sl < 4 ? nx0 : nx1, b), X.a, X.bn), tfx = fmaf(q8(sl < 4 ? fx0 : fx1, b), X.a, X.bf);
            const float tny = fmaf(q8(sl < 4 ? ny0 : ny1, b), Y.a, Y.bn), tfy = fmaf(q8(sl < 4 ? fy0 : fy1, b), Y.a, Y.bf);
            const float tnz = fmaf(q8(sl < 4 ? nz0 : nz1, b), Z.a, Z.bn), tfz = fmaf(q8(sl < 4 ? fz0 : fz1, b), Z.a, Z.bf);
            const float tn = fmax3(tnx, tny, fmaxf(tnz, 0.0f));
            const float tf = fmin3(tfx, tfy, fminf(tfz, best)) * widen;
            hits |= (tn <= tf ? 1u : 0u) << sl;
        }
        hits &= valid;
        // triangles of the hit leaves of this node
        uint32_t leaves = hits & ~imask, tbits = 0;
        while (leaves) {
            const uint32_t sl = __ffs(leaves) - 1;
            leaves &= leaves - 1;
            const uint32_t meta = ((sl < 4 ? w1.z : w1.w) >> (8 * (sl & 3))) & 0xFFu;
            tbits |= ((1u << (meta >> 5)) - 1u) << (meta & 31u);
        }
        while (tbits) {
            const uint32_t k = __ffs(tbits) - 1;
            tbits &= tbits - 1;
            const uint32_t ti = tri_base + k;
            const float4 t0 = __ldg(&tris[3 * ti + 0]);
            const float4 t1 = __ldg(&tris[3 * ti + 1]);
            const float4 t2 = __ldg(&tris[3 * ti + 2]);
            if (COUNT) cnt.tris++;
            float tt, U, V, W, det;
            if (wt_test(r, ld3(t0), ld3(t1), ld3(t2), tt, U, V, W, det)) {
                const uint32_t id = __float_as_uint(t0.w);
                if (any) {
                    if (tt <= tmax) { h.t = tt; h.id = id; return; }
                } else if (tt < h.t || (tt == h.t && id < h.id)) {
                    h.t = tt; h.id = id; h.U = U; h.V = V; h.W = W; h.det = det;
                    best = tt;
                }
            }
        }
        // next node: the nearest remaining hit child of this node, else of the stacked groups
        uint32_t pending = octant_order(hits & imask, oct), base = child_base, im = imask;
        if (!pending) {
            if (sp == 0) return;
            const uint2 g = stack[--sp];
            base = g.x; pending = g.y & 0xFFu; im = g.y >> 8;
        }
        const uint32_t k = __ffs(pending) - 1;
        pending &= pending - 1;
        const uint32_t slot = oct ^ k;
        node = base + __popc(im & ((1u << slot) - 1u));
        if (pending) {
            if (sp >= kStack8) { err |= kErrStack; return; }
            stack[sp++] = make_uint2(base, pending | (im << 8));
        }
    }
}

template <bool ANY, bool COUNT>
__device__ __forceinline__ void traverse8(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                          const WRay& r, float tmax, HitOut& h, uint32_t& err, Counters& cnt,
                                          uint32_t cap) {
    traverse8_rt<COUNT>(nodes, tris, r, tmax, ANY, h, err, cnt, cap);
}

// Dispatch on the node layout (2: binary, occlusion only; 4: wide; 8: compressed 8-wide).  `cap`: traversal steps
// per ray before the ray gives up and sets kErrIter.  UNIT: the ray's direction is normalised.
template <int LAYOUT, bool ANY, bool COUNT, bool UNIT = true>
__device__ __forceinline__ void traverse_any_layout(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                    const WRay& r, float tmax, HitOut& h, uint32_t& err, Counters& cnt,
                                                    uint32_t cap) {
    static_assert(LAYOUT != 2 || ANY, "closest hits walk the wide nodes");
    if (LAYOUT == 8) traverse8<ANY, COUNT>(nodes, tris, r, tmax, h, err, cnt, cap);
    else if (LAYOUT == 4) traverse4_rt<COUNT, UNIT>(nodes, tris, r, tmax, ANY, h, err, cnt, cap);
    else occluded2<COUNT>(reinterpret_cast<const float4*>(nodes), tris, r, tmax, h, err, cnt, cap);
}

}  // namespace vgbd
