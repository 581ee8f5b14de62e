// Closest-hit and any-hit traversal of the 4-wide BVH.
//
// By default the box and triangle tests repeat the reference's arithmetic
// exactly (no fused multiply-add): the slab test of BoundingBox3D::intersect
// (libSLR/BasicTypes/BoundingBox3D.h:100-116) on the SBVH's own boxes, and
// the Moller-Trumbore test of TriangleSurfaceShape::intersect
// (libSLR/SurfaceShape/TriangleSurfaceShape.cpp:205-257), including its
// inclusive [tmin, tmax] acceptance.  The wide nodes only skip the SBVH's
// intermediate boxes, which contain their children's boxes, so every
// triangle the reference would test is still tested.  With
// DevScene::watertight the triangle test is the watertight one below.
#pragma once
#include "device_common.cuh"

namespace slrgpu {

struct Hit {
    float t, b1, b2;
    uint32_t prim;
};

constexpr uint32_t kNoHit = 0xffffffffu;
constexpr int kTraceStack = 96;

// Moller-Trumbore; returns true and t/b1/b2 when the triangle is hit within [tmin, tmax].
__device__ __forceinline__ bool mtIntersect(const TriFrag &f, V3 org, V3 dir, float tmin, float tmax,
                                            float* tOut, float* b1Out, float* b2Out) {
    V3 e1 = V3{f.e1x, f.e1y, f.e1z};
    V3 e2 = V3{f.e2x, f.e2y, f.e2z};
    V3 p = rn_cross(dir, e2);
    float det = rn_dot(e1, p);
    if (det == 0.0f) return false;
    float invDet = __frcp_rn(det);   // 1 / det, correctly rounded as the division
    V3 d = rn_sub(org, V3{f.v0x, f.v0y, f.v0z});
    float b1 = __fmul_rn(rn_dot(d, p), invDet);
    if (b1 < 0.0f || b1 > 1.0f) return false;
    V3 q = rn_cross(d, e1);
    float b2 = __fmul_rn(rn_dot(dir, q), invDet);
    if (b2 < 0.0f || __fadd_rn(b1, b2) > 1.0f) return false;
    float tt = __fmul_rn(rn_dot(e2, q), invDet);
    if (tt < tmin || tt > tmax) return false;
    *tOut = tt;
    *b1Out = b1;
    *b2Out = b2;
    return true;
}

// Watertight ray-triangle test (Woop, Benthin and Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2013): vertices translated to the ray
// origin and sheared so the ray runs along +z; the 2-D edge functions are
// exact in sign for edges shared by two triangles (recomputed in double when
// one is zero), so a ray never slips between adjacent triangles.  Uses the
// vertices as given (not v0 + edge).  b1, b2 are the weights of v1 and v2, t
// is accepted in [tmin, tmax] as the reference's test does.
struct WtRay {
    int kx, ky, kz;
    float sx, sy, sz;
    V3 org;
};

__device__ __forceinline__ WtRay wtSetup(V3 org, V3 dir) {
    const float d[3] = {dir.x, dir.y, dir.z};
    const float ax = fabsf(dir.x), ay = fabsf(dir.y), az = fabsf(dir.z);
    int kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz == 2 ? 0 : kz + 1;
    int ky = kx == 2 ? 0 : kx + 1;
    float dz = kz == 0 ? d[0] : (kz == 1 ? d[1] : d[2]);
    if (dz < 0.0f) { int tmp = kx; kx = ky; ky = tmp; }
    const float dx = kx == 0 ? d[0] : (kx == 1 ? d[1] : d[2]);
    const float dy = ky == 0 ? d[0] : (ky == 1 ? d[1] : d[2]);
    WtRay r;
    r.kx = kx; r.ky = ky; r.kz = kz;
    r.sx = dx / dz;
    r.sy = dy / dz;
    r.sz = 1.0f / dz;
    r.org = org;
    return r;
}

__device__ __forceinline__ float comp(V3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }

__device__ __forceinline__ bool wtIntersect(const float4* __restrict__ wv, uint32_t i, const WtRay &r, float tmin,
                                            float tmax, float* tOut, float* b1Out, float* b2Out, uint32_t* prim) {
    const float4 p0 = __ldg(wv + 3 * (size_t)i), p1 = __ldg(wv + 3 * (size_t)i + 1), p2 = __ldg(wv + 3 * (size_t)i + 2);
    const V3 A = V3{p0.x, p0.y, p0.z} - r.org, B = V3{p1.x, p1.y, p1.z} - r.org, C = V3{p2.x, p2.y, p2.z} - r.org;
    const float Az = comp(A, r.kz), Bz = comp(B, r.kz), Cz = comp(C, r.kz);
    const float Ax = comp(A, r.kx) - r.sx * Az, Ay = comp(A, r.ky) - r.sy * Az;
    const float Bx = comp(B, r.kx) - r.sx * Bz, By = comp(B, r.ky) - r.sy * Bz;
    const float Cx = comp(C, r.kx) - r.sx * Cz, Cy = comp(C, r.ky) - r.sy * Cz;
    // Each product rounded on its own (no fused multiply-add): the edge
    // function of an edge shared by two triangles must come out exactly
    // negated in the neighbour, which a contraction would break.
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        U = (float)__dsub_rn(__dmul_rn(Cx, By), __dmul_rn(Cy, Bx));
        V = (float)__dsub_rn(__dmul_rn(Ax, Cy), __dmul_rn(Ay, Cx));
        W = (float)__dsub_rn(__dmul_rn(Bx, Ay), __dmul_rn(By, Ax));
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = U + V + W;
    if (det == 0.0f) return false;
    const float T = U * (r.sz * Az) + V * (r.sz * Bz) + W * (r.sz * Cz);
    const float inv = 1.0f / det;
    const float t = T * inv;
    if (!(t >= tmin && t <= tmax)) return false;
    *tOut = t;
    *b1Out = V * inv;
    *b2Out = W * inv;
    *prim = __float_as_uint(p0.w);
    return true;
}

// Slab test; returns the entry distance (dist0) or +inf when rejected.
// `robust` widens each slab's exit distance by 1 + 2 gamma_3 (Ize, "Robust
// BVH Ray Traversal", JCGT 2013) so that rounding cannot reject a box the
// ray only grazes at a face, edge or corner; the watertight triangle test
// needs it, the reference's arithmetic does not have it.
template <bool ROBUST>
__device__ __forceinline__ float slabTest(float lox, float hix, float loy, float hiy, float loz, float hiz,
                                          V3 org, V3 inv, float tmin, float tmax) {
    float d0 = tmin, d1 = tmax;
    float tn = __fmul_rn(__fsub_rn(lox, org.x), inv.x), tf = __fmul_rn(__fsub_rn(hix, org.x), inv.x);
    if (tn > tf) { float s = tn; tn = tf; tf = s; }
    if (ROBUST) tf = __fmul_rn(tf, 1.0000008f);
    d0 = tn > d0 ? tn : d0;
    d1 = tf < d1 ? tf : d1;
    tn = __fmul_rn(__fsub_rn(loy, org.y), inv.y); tf = __fmul_rn(__fsub_rn(hiy, org.y), inv.y);
    if (tn > tf) { float s = tn; tn = tf; tf = s; }
    if (ROBUST) tf = __fmul_rn(tf, 1.0000008f);
    d0 = tn > d0 ? tn : d0;
    d1 = tf < d1 ? tf : d1;
    tn = __fmul_rn(__fsub_rn(loz, org.z), inv.z); tf = __fmul_rn(__fsub_rn(hiz, org.z), inv.z);
    if (tn > tf) { float s = tn; tn = tf; tf = s; }
    if (ROBUST) tf = __fmul_rn(tf, 1.0000008f);
    d0 = tn > d0 ? tn : d0;
    d1 = tf < d1 ? tf : d1;
    return (d0 > d1) ? __int_as_float(0x7f800000) : d0;
}

#ifndef SLRGPU_MINMAX_SLABS
#define SLRGPU_MINMAX_SLABS 1
#endif

struct StackEntry {
    uint32_t node;
    float tnear;
};

// The walk's stack: a thread's own array in local memory, or its first S
// entries in shared memory ([entry][thread], blocks of 256) and the rest local.
template <typename T>
struct LocalStack {
    T rest[kTraceStack];
    __device__ __forceinline__ void put(int i, T e) { rest[i] = e; }
    __device__ __forceinline__ T get(int i) const { return rest[i]; }
};
template <typename T, int S>
struct SharedStack {
    T* top;
    T rest[kTraceStack - S];
    __device__ __forceinline__ explicit SharedStack(T* shared) : top(shared + threadIdx.x) {}
    __device__ __forceinline__ void put(int i, T e) {
        if (i < S) top[i * 256] = e;
        else rest[i - S] = e;
    }
    __device__ __forceinline__ T get(int i) const { return i < S ? top[i * 256] : rest[i - S]; }
};

// A node visit is bound by its instructions (the walk issues on two thirds of
// its cycles) and by the lines its lanes' loads touch.  Loading a node as
// three 32-byte halves of its box planes and its child words instead of seven
// 16-byte parts, testing two boxes per packed instruction and ordering the
// children without carrying their numbers took 1,000,003 incoherent closest-hit
// queries on 24k triangles from 489 to 456 us and 4 Mi any-hit queries on 176k
// triangles from 1697 to 1528 us (without the loads 476 and 1675 us, without the
// packed tests 465 and 1561 us).

// 32 bytes of read-only global memory in one load (p 32-byte aligned).
__device__ __forceinline__ void ldg256(const float4* p, float4 &a, float4 &b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// Two single-precision operations in one instruction, each rounded as the
// scalar one.
struct F2 { uint64_t v; };
__device__ __forceinline__ F2 f2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void f2get(F2 a, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 f2add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// slabTest as min/max operations for two boxes at once, the twelve differences
// and products of each pair packed two to an instruction, for rays whose
// inverse direction is finite in every axis: then no product is NaN, the
// compare-and-swap of each slab's two distances is their min and max, and the running entry and
// exit distances are a max and a min (the order of the axes does not
// change a max or a min), so every distance and decision equals slabTest's
// (up to the sign of a zero, which no comparison sees).  A zero direction
// component makes (plane - origin) * inv NaN on a plane through the origin,
// where slabTest's comparisons decide differently from min/max; such rays
// take slabTest.
template <bool ROBUST>
__device__ __forceinline__ void slabTestMinMax2(F2 lox, F2 hix, F2 loy, F2 hiy, F2 loz, F2 hiz, V3 org, V3 inv,
                                                float tmin, float tmax, float &tn0, float &tn1) {
    // plane - origin as plane + (-origin): the same rounding
    const F2 ox = f2(-org.x, -org.x), oy = f2(-org.y, -org.y), oz = f2(-org.z, -org.z);
    const F2 ix = f2(inv.x, inv.x), iy = f2(inv.y, inv.y), iz = f2(inv.z, inv.z);
    float ax[2], bx[2], ay[2], by[2], az[2], bz[2];
    f2get(f2mul(f2add(lox, ox), ix), ax[0], ax[1]);
    f2get(f2mul(f2add(hix, ox), ix), bx[0], bx[1]);
    f2get(f2mul(f2add(loy, oy), iy), ay[0], ay[1]);
    f2get(f2mul(f2add(hiy, oy), iy), by[0], by[1]);
    f2get(f2mul(f2add(loz, oz), iz), az[0], az[1]);
    f2get(f2mul(f2add(hiz, oz), iz), bz[0], bz[1]);
    float r[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        float fx = fmaxf(ax[k], bx[k]), fy = fmaxf(ay[k], by[k]), fz = fmaxf(az[k], bz[k]);
        if (ROBUST) {
            fx = __fmul_rn(fx, 1.0000008f);
            fy = __fmul_rn(fy, 1.0000008f);
            fz = __fmul_rn(fz, 1.0000008f);
        }
        const float d0 = fmaxf(fmaxf(fminf(ax[k], bx[k]), fminf(ay[k], by[k])), fmaxf(fminf(az[k], bz[k]), tmin));
        const float d1 = fminf(fminf(fx, fy), fminf(fz, tmax));
        r[k] = (d0 > d1) ? __int_as_float(0x7f800000) : d0;
    }
    tn0 = r[0];
    tn1 = r[1];
}

// Box test of the 4 children of a node; returns the hit mask and entry distances.
template <bool ROBUST>
__device__ __forceinline__ uint32_t testChildren(const BvhNode* __restrict__ nodes, uint32_t ni, V3 org, V3 inv,
                                                 float tmin, float tmax, float tn[kBvhWidth],
                                                 uint32_t ch[kBvhWidth], bool minmax = false) {
    // 128-bit loads: Q float4 per coordinate array, then the child words
    constexpr int Q = kBvhWidth / 4;
    const float4* np = reinterpret_cast<const float4*>(nodes + ni);
    uint32_t mask = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        float4 lx, hx, ly, hy, lz, hz;
        if constexpr (kBvhWidth == 4) {
            ldg256(np, lx, hx);
            ldg256(np + 2, ly, hy);
            ldg256(np + 4, lz, hz);
        } else {
            lx = __ldg(np + 0 * Q + q), hx = __ldg(np + 1 * Q + q), ly = __ldg(np + 2 * Q + q);
            hy = __ldg(np + 3 * Q + q), lz = __ldg(np + 4 * Q + q), hz = __ldg(np + 5 * Q + q);
        }
        const uint4 c = __ldg(reinterpret_cast<const uint4*>(np + 6 * Q) + q);
        const float lxa[4] = {lx.x, lx.y, lx.z, lx.w}, hxa[4] = {hx.x, hx.y, hx.z, hx.w};
        const float lya[4] = {ly.x, ly.y, ly.z, ly.w}, hya[4] = {hy.x, hy.y, hy.z, hy.w};
        const float lza[4] = {lz.x, lz.y, lz.z, lz.w}, hza[4] = {hz.x, hz.y, hz.z, hz.w};
        const uint32_t ca[4] = {c.x, c.y, c.z, c.w};
        if (SLRGPU_MINMAX_SLABS && minmax) {
            slabTestMinMax2<ROBUST>(f2(lx.x, lx.y), f2(hx.x, hx.y), f2(ly.x, ly.y), f2(hy.x, hy.y), f2(lz.x, lz.y),
                                    f2(hz.x, hz.y), org, inv, tmin, tmax, tn[4 * q], tn[4 * q + 1]);
            slabTestMinMax2<ROBUST>(f2(lx.z, lx.w), f2(hx.z, hx.w), f2(ly.z, ly.w), f2(hy.z, hy.w), f2(lz.z, lz.w),
                                    f2(hz.z, hz.w), org, inv, tmin, tmax, tn[4 * q + 2], tn[4 * q + 3]);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int i = 4 * q + k;
                ch[i] = ca[k];
                if (ch[i] != kChildEmpty && tn[i] != __int_as_float(0x7f800000)) mask |= 1u << i;
            }
            continue;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = 4 * q + k;
            ch[i] = ca[k];
            tn[i] = slabTest<ROBUST>(lxa[k], hxa[k], lya[k], hya[k], lza[k], hza[k], org, inv, tmin, tmax);
            if (ch[i] != kChildEmpty && tn[i] != __int_as_float(0x7f800000)) mask |= 1u << i;
        }
    }
    return mask;
}

// Orders the hit children of a node near to far (ties in child order) with a
// sorting network on registers (5 comparators for 4 children, Batcher's 19
// for 8); missed children sort last at +inf.  Pushes all but the nearest,
// far to near, and returns the nearest.
template <class STACK>
__device__ __forceinline__ uint32_t orderChildren(uint32_t mask, const float tn[kBvhWidth],
                                                  const uint32_t ch[kBvhWidth], STACK &stack, int &sp,
                                                  bool &ok) {
    if constexpr (kBvhWidth == 4) {
        // The same network without carrying the child numbers.  Comparing
        // (0,1), (2,3), then (0,2), (1,3) leaves a tie's lower child on the
        // left without a swap.  In the last comparison (1,2) the left element
        // is the lower child of a tie only if neither comparison before it
        // swapped; after a swap a tie swaps too.
        const float inf = __int_as_float(0x7f800000);
        float t0 = (mask & 1u) ? tn[0] : inf, t1 = (mask & 2u) ? tn[1] : inf;
        float t2 = (mask & 4u) ? tn[2] : inf, t3 = (mask & 8u) ? tn[3] : inf;
        uint32_t c0 = ch[0], c1 = ch[1], c2 = ch[2], c3 = ch[3];
#define SLRGPU_CSWAP(s, a, b)                                        \
    {                                                                \
        const float ta = s ? t##b : t##a, tb = s ? t##a : t##b;      \
        const uint32_t ca = s ? c##b : c##a, cb = s ? c##a : c##b;   \
        t##a = ta; t##b = tb; c##a = ca; c##b = cb;                  \
    }
        const bool s01 = t1 < t0;
        SLRGPU_CSWAP(s01, 0, 1)
        const bool s23 = t3 < t2;
        SLRGPU_CSWAP(s23, 2, 3)
        const bool s02 = t2 < t0;
        SLRGPU_CSWAP(s02, 0, 2)
        const bool s13 = t3 < t1;
        SLRGPU_CSWAP(s13, 1, 3)
        const bool s12 = t2 < t1 || ((s02 || s13) && t2 == t1);
        SLRGPU_CSWAP(s12, 1, 2)
#undef SLRGPU_CSWAP
        const int n = __popc(mask);
        if (sp + n - 1 <= kTraceStack) {
            if (n > 3) stack.put(sp++, StackEntry{c3, t3});
            if (n > 2) stack.put(sp++, StackEntry{c2, t2});
            if (n > 1) stack.put(sp++, StackEntry{c1, t1});
        } else {   // the farthest that fit
            if (n > 3 && sp < kTraceStack) stack.put(sp++, StackEntry{c3, t3});
            if (n > 2 && sp < kTraceStack) stack.put(sp++, StackEntry{c2, t2});
            if (n > 1 && sp < kTraceStack) stack.put(sp++, StackEntry{c1, t1});
            ok = false;
        }
        return c0;
    }
    float t[kBvhWidth];
    uint32_t c[kBvhWidth], k[kBvhWidth];
#pragma unroll
    for (int i = 0; i < kBvhWidth; ++i) {
        t[i] = ((mask >> i) & 1u) ? tn[i] : __int_as_float(0x7f800000);
        c[i] = ch[i];
        k[i] = (uint32_t)i;
    }
#define SLRGPU_CSWAP(a, b)                                                           \
    if (t[b] < t[a] || (t[b] == t[a] && k[b] < k[a])) {                              \
        float tt = t[a]; t[a] = t[b]; t[b] = tt;                                     \
        uint32_t cc = c[a]; c[a] = c[b]; c[b] = cc;                                  \
        uint32_t kk = k[a]; k[a] = k[b]; k[b] = kk;                                  \
    }
    if constexpr (kBvhWidth == 4) {
        SLRGPU_CSWAP(0, 1) SLRGPU_CSWAP(2, 3) SLRGPU_CSWAP(0, 2) SLRGPU_CSWAP(1, 3) SLRGPU_CSWAP(1, 2)
    } else {
        SLRGPU_CSWAP(0, 1) SLRGPU_CSWAP(2, 3) SLRGPU_CSWAP(4, 5) SLRGPU_CSWAP(6, 7)
        SLRGPU_CSWAP(0, 2) SLRGPU_CSWAP(1, 3) SLRGPU_CSWAP(4, 6) SLRGPU_CSWAP(5, 7)
        SLRGPU_CSWAP(1, 2) SLRGPU_CSWAP(5, 6)
        SLRGPU_CSWAP(0, 4) SLRGPU_CSWAP(1, 5) SLRGPU_CSWAP(2, 6) SLRGPU_CSWAP(3, 7)
        SLRGPU_CSWAP(2, 4) SLRGPU_CSWAP(3, 5)
        SLRGPU_CSWAP(1, 2) SLRGPU_CSWAP(3, 4) SLRGPU_CSWAP(5, 6)
    }
#undef SLRGPU_CSWAP
    const int n = __popc(mask);
#pragma unroll
    for (int i = kBvhWidth - 1; i >= 1; --i) {
        if (i < n) {
            if (sp < kTraceStack) stack.put(sp++, StackEntry{c[i], t[i]});
            else ok = false;
        }
    }
    return c[0];
}

// WIDE: the first half as one 32-byte load.  The any-hit walk gains from it (4 Mi
// queries on 176k triangles 1530 us with three 16-byte loads of a 48-byte
// record, 1469 us so); the closest-hit walk, short of registers, loses 2 %.
template <bool WIDE>
__device__ __forceinline__ TriFrag loadFrag(const TriFrag* __restrict__ frags, uint32_t i) {
    const float4* p = reinterpret_cast<const float4*>(frags + i);
    float4 a, b;
    if (WIDE) {
        ldg256(p, a, b);
    } else {
        a = __ldg(p);
        b = __ldg(p + 1);
    }
    const float4 c = __ldg(p + 2);
    TriFrag f;
    f.v0x = a.x; f.v0y = a.y; f.v0z = a.z; f.prim = __float_as_uint(a.w);
    f.e1x = b.x; f.e1y = b.y; f.e1z = b.z; f.pad0 = 0;
    f.e2x = c.x; f.e2y = c.y; f.e2z = c.z; f.pad1 = 0;
    return f;
}

// A closest-hit walk over [tmin, tmax] that can stop after a number of node
// or leaf visits and resume later: the wave kernels give a lane a new ray as
// soon as its walk ends, instead of leaving it idle until the longest walk of
// its warp is done.  Nodes and triangles are visited in the order of an
// uninterrupted walk, so the hit is the same.  WT: the watertight triangle
// test with conservative box tests.
template <bool WT>
struct ClosestWalk {
    V3 org, dir, inv;
    WtRay wr;
    float tmin, tmax;
    Hit hit;
    uint32_t cur;
    int sp;
    bool ok;   // false after a stack overflow (the hit found so far is kept)
    bool minmax;   // finite inverse direction: slabTestMinMax2

    // Returns true when the walk has already ended (an empty scene).
    __device__ __forceinline__ bool begin(const DevScene &sc, V3 o, V3 d, float t0, float t1) {
        hit.prim = kNoHit;
        hit.t = __int_as_float(0x7f800000);
        hit.b1 = hit.b2 = 0.0f;
        org = o;
        dir = d;
        inv = V3{__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z)};
        minmax = isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z);
        if (WT) wr = wtSetup(o, d);
        tmin = t0;
        tmax = t1;
        cur = 0;
        sp = 0;
        ok = true;
        return sc.numPrims == 0;
    }

    // At most `visits` node or leaf visits; returns true when the walk has ended.
    template <class STACK>
    __device__ __forceinline__ bool advance(const DevScene &sc, STACK &stack, int visits) {
        for (int v = 0; v < visits; ++v) {
            if (!(cur & kLeafBit)) {
                float tn[kBvhWidth];
                uint32_t ch[kBvhWidth];
                const uint32_t mask = testChildren<WT>(sc.nodes, cur, org, inv, tmin, tmax, tn, ch, minmax);
                if (mask != 0) {
                    cur = orderChildren(mask, tn, ch, stack, sp, ok);
                    continue;
                }
            } else {
                const uint32_t first = cur & kLeafFirstMask;
                const uint32_t count = ((cur >> kLeafCountShift) & 0x1f) + 1;
                for (uint32_t i = 0; i < count; ++i) {
                    float t, b1, b2;
                    uint32_t prim;
                    bool h;
                    if (WT) {
                        h = wtIntersect(sc.wtVerts, first + i, wr, tmin, tmax, &t, &b1, &b2, &prim);
                    } else {
                        TriFrag f = loadFrag<false>(sc.frags, first + i);
                        h = mtIntersect(f, org, dir, tmin, tmax, &t, &b1, &b2);
                        prim = f.prim;
                    }
                    if (h) {
                        tmax = t;
                        hit.t = t;
                        hit.b1 = b1;
                        hit.b2 = b2;
                        hit.prim = prim;
                    }
                }
            }
            // the nearest pushed node the ray can still reach
            for (;;) {
                if (sp == 0) return true;
                const StackEntry e = stack.get(--sp);
                if (e.tnear <= tmax) {
                    cur = e.node;
                    break;
                }
            }
        }
        return false;
    }
};

// Closest hit over [tmin, tmax] in one go.  Returns false on stack overflow
// (the hit found so far is still reported).
template <bool WT>
__device__ __forceinline__ bool traceClosestT(const DevScene &sc, V3 org, V3 dir, float tmin, float tmax, Hit* hit) {
    LocalStack<StackEntry> stack;
    ClosestWalk<WT> w;
    if (!w.begin(sc, org, dir, tmin, tmax))
        while (!w.advance(sc, stack, 1 << 30)) {
        }
    *hit = w.hit;
    return w.ok;
}

__device__ __forceinline__ bool traceClosest(const DevScene &sc, V3 org, V3 dir, float tmin, float tmax, Hit* hit) {
    return sc.watertight ? traceClosestT<true>(sc, org, dir, tmin, tmax, hit)
                         : traceClosestT<false>(sc, org, dir, tmin, tmax, hit);
}

// An any-hit walk over [tmin, tmax] that can stop and resume like
// ClosestWalk; `occluded` holds the answer once the walk has ended.
template <bool WT>
struct AnyWalk {
    V3 org, dir, inv;
    WtRay wr;
    float tmin, tmax;
    uint32_t cur;
    int sp;
    bool occluded;
    bool minmax;

    __device__ __forceinline__ bool begin(const DevScene &sc, V3 o, V3 d, float t0, float t1) {
        org = o;
        dir = d;
        inv = V3{__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z)};
        minmax = isfinite(inv.x) && isfinite(inv.y) && isfinite(inv.z);
        if (WT) wr = wtSetup(o, d);
        tmin = t0;
        tmax = t1;
        cur = 0;
        sp = 0;
        occluded = false;
        return sc.numPrims == 0;
    }

    template <class STACK>
    __device__ __forceinline__ bool advance(const DevScene &sc, STACK &stack, int visits) {
        for (int v = 0; v < visits; ++v) {
            if (!(cur & kLeafBit)) {
                float tn[kBvhWidth];
                uint32_t ch[kBvhWidth];
                const uint32_t mask = testChildren<WT>(sc.nodes, cur, org, inv, tmin, tmax, tn, ch, minmax);
                bool have = false;
                uint32_t next = 0;
#pragma unroll
                for (int k = 0; k < kBvhWidth; ++k) {
                    if (mask & (1u << k)) {
                        if (!have) { next = ch[k]; have = true; }
                        else if (sp < kTraceStack) stack.put(sp++, ch[k]);
                    }
                }
                if (have) {
                    cur = next;
                    continue;
                }
            } else {
                const uint32_t first = cur & kLeafFirstMask;
                const uint32_t count = ((cur >> kLeafCountShift) & 0x1f) + 1;
                for (uint32_t i = 0; i < count; ++i) {
                    float t, b1, b2;
                    bool h;
                    if (WT) {
                        uint32_t prim;
                        h = wtIntersect(sc.wtVerts, first + i, wr, tmin, tmax, &t, &b1, &b2, &prim);
                    } else {
                        TriFrag f = loadFrag<true>(sc.frags, first + i);
                        h = mtIntersect(f, org, dir, tmin, tmax, &t, &b1, &b2);
                    }
                    if (h) {
                        occluded = true;
                        return true;
                    }
                }
            }
            if (sp == 0) return true;
            cur = stack.get(--sp);
        }
        return false;
    }
};

// Any hit over [tmin, tmax]: true when the segment is occluded.
template <bool WT>
__device__ __forceinline__ bool traceAnyT(const DevScene &sc, V3 org, V3 dir, float tmin, float tmax) {
    LocalStack<uint32_t> stack;
    AnyWalk<WT> w;
    if (w.begin(sc, org, dir, tmin, tmax)) return false;
    while (!w.advance(sc, stack, 1 << 30)) {
    }
    return w.occluded;
}

__device__ __forceinline__ bool traceAny(const DevScene &sc, V3 org, V3 dir, float tmin, float tmax) {
    return sc.watertight ? traceAnyT<true>(sc, org, dir, tmin, tmax) : traceAnyT<false>(sc, org, dir, tmin, tmax);
}

// ---------------------------------------------------------------------------
// Dynamic ray fetch of the wave kernels
// ---------------------------------------------------------------------------
#ifndef SLRGPU_TRACE_REFILL_LANES
#define SLRGPU_TRACE_REFILL_LANES 8
#endif
#ifndef SLRGPU_TRACE_REFILL_VISITS
#define SLRGPU_TRACE_REFILL_VISITS 16
#endif
static_assert(SLRGPU_TRACE_REFILL_LANES >= 1 && SLRGPU_TRACE_REFILL_LANES <= 32, "a warp has 32 lanes");
// Stack entries of a closest-hit walk in shared memory: lanes at different
// depths store to as many lines of local memory, but to different banks of
// shared memory.  1,000,003 incoherent queries on 24k triangles 456 us without,
// 448, 441, 440 and 441 with 4, 8, 12 and 16 entries.  The any-hit walk's
// 4-byte entries stay local (4 Mi queries on 176k triangles 1528 us, 1557 with
// 12 entries in shared memory: the L1 it takes counts for more).
constexpr int kSharedStackEntries = 8;
using ClosestStack = SharedStack<StackEntry, kSharedStackEntries>;

// The refill step of a warp: when at least SLRGPU_TRACE_REFILL_LANES lanes
// are idle and the queue is not drained, the idle lanes take the next queue
// entries (*slot = entry index, or n when there is none left).  Returns
// whether this lane got one.  Called by all 32 lanes.
__device__ __forceinline__ bool refillLanes(bool live, uint32_t* cursor, uint32_t n, bool &drained, uint32_t* slot) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t idle = __ballot_sync(0xffffffffu, !live);
    if (drained || (uint32_t)__popc(idle) < SLRGPU_TRACE_REFILL_LANES) return false;
    const int leader = __ffs(idle) - 1;
    uint32_t base = 0;
    if ((int)lane == leader) base = atomicAdd(cursor, (uint32_t)__popc(idle));
    base = __shfl_sync(0xffffffffu, base, leader);
    drained = base + (uint32_t)__popc(idle) >= n;
    if (live) return false;
    *slot = base + (uint32_t)__popc(idle & ((1u << lane) - 1));
    return *slot < n;
}

}  // namespace slrgpu
