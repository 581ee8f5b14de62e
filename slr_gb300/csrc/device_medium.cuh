// Heterogeneous medium on the device: density-grid lookups, the super-voxel
// 3-D DDA with a cubic majorant per cell and regula-falsi free-path solve,
// delta tracking for scattering and ratio tracking for transmittance.  The
// arithmetic follows DensityGridMediumDistribution
// (libSLR/MediumDistribution/DensityGridMediumDistribution.cpp:16-744) and the
// single-medium case of MediumObjectAggregate::interact / evaluateTransmittance
// (libSLR/Core/medium_object.cpp:287-402).
#pragma once
#include "device_common.cuh"

namespace slrgpu {

__device__ __forceinline__ bool outsideUnit(V3 p) {
    return p.x < 0 || p.y < 0 || p.z < 0 || p.x > 1 || p.y > 1 || p.z > 1;
}

__device__ __forceinline__ float trilinearGrid(const float* __restrict__ g, uint32_t nx, uint32_t ny, uint32_t nz, V3 p) {
    uint32_t lx = min((uint32_t)(p.x * (nx - 1)), nx - 1), ux = min(lx + 1, nx - 1);
    uint32_t ly = min((uint32_t)(p.y * (ny - 1)), ny - 1), uy = min(ly + 1, ny - 1);
    uint32_t lz = min((uint32_t)(p.z * (nz - 1)), nz - 1), uz = min(lz + 1, nz - 1);
    float wux = p.x * (nx - 1) - lx, wlx = 1 - wux;
    float wuy = p.y * (ny - 1) - ly, wly = 1 - wuy;
    float wuz = p.z * (nz - 1) - lz, wlz = 1 - wuz;
    const size_t sl = (size_t)nx * ny;
    const float* zl = g + sl * lz;
    const float* zu = g + sl * uz;
    return __ldg(zl + nx * ly + lx) * wlz * wly * wlx + __ldg(zl + nx * ly + ux) * wlz * wly * wux +
           __ldg(zl + nx * uy + lx) * wlz * wuy * wlx + __ldg(zl + nx * uy + ux) * wlz * wuy * wux +
           __ldg(zu + nx * ly + lx) * wuz * wly * wlx + __ldg(zu + nx * ly + ux) * wuz * wly * wux +
           __ldg(zu + nx * uy + lx) * wuz * wuy * wlx + __ldg(zu + nx * uy + ux) * wuz * wuy * wux;
}

// calcDensity (DensityGridMediumDistribution.cpp:369-395).
__device__ __forceinline__ float mediumDensity(const DevMedium &m, V3 param) {
    if (outsideUnit(param)) return 0.0f;
    return trilinearGrid(m.density, m.nx, m.ny, m.nz, param);
}

// calcDensityInSuperVoxels (DensityGridMediumDistribution.cpp:16-43).
__device__ __forceinline__ float mediumCoarseDensity(const DevMedium &m, V3 param) {
    if (outsideUnit(param)) return 0.0f;
    float d = trilinearGrid(m.superVoxels, m.svx, m.svy, m.svz, param);
    uint32_t lx = min((uint32_t)(param.x * (m.svx - 1)), m.svx - 1);
    uint32_t ly = min((uint32_t)(param.y * (m.svy - 1)), m.svy - 1);
    uint32_t lz = min((uint32_t)(param.z * (m.svz - 1)), m.svz - 1);
    uint32_t cell = (m.svx - 1) * (m.svy - 1) * min(lz, m.svz - 2) + (m.svx - 1) * min(ly, m.svy - 2) + min(lx, m.svx - 2);
    return d + m.maxDiff[cell];
}

// Position in the medium's unit cube.  The divisions of the reference become
// multiplications by reciprocals computed once on the host (results differ
// in the last bit; the walks are issue-bound and an IEEE division is a
// sequence of instructions).
__device__ __forceinline__ V3 mediumLocal(const DevMedium &m, V3 p) {
    return V3{(p.x - m.bmin[0]) * m.invExtent[0], (p.y - m.bmin[1]) * m.invExtent[1],
              (p.z - m.bmin[2]) * m.invExtent[2]};
}

constexpr float kThird = 1.0f / 3.0f;

__device__ __forceinline__ bool mediumContains(const DevMedium &m, V3 p) {
    return p.x >= m.bmin[0] && p.x < m.bmax[0] && p.y >= m.bmin[1] && p.y < m.bmax[1] && p.z >= m.bmin[2] &&
           p.z < m.bmax[2];
}

// BoundingBox3D::intersectBoundary (BoundingBox3D.h:119-144).
__device__ __forceinline__ bool mediumIntersectBoundary(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                                       float* dist, bool* enter) {
    float d0 = -__int_as_float(0x7f800000), d1 = __int_as_float(0x7f800000);
    const float o[3] = {org.x, org.y, org.z}, d[3] = {dir.x, dir.y, dir.z};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        float inv = 1.0f / d[i];
        float tn = (m.bmin[i] - o[i]) * inv, tf = (m.bmax[i] - o[i]) * inv;
        if (tn > tf) { float s = tn; tn = tf; tf = s; }
        d0 = tn > d0 ? tn : d0;
        d1 = tf < d1 ? tf : d1;
        if (d0 > d1) return false;
    }
    if (mediumContains(m, org + dmin * dir)) {
        *dist = d1;
        *enter = false;
        return d1 >= dmin && d1 < dmax;
    }
    *dist = d0;
    *enter = true;
    return d0 >= dmin && d0 < dmax;
}

// ---- super-voxel traversal -------------------------------------------------
// The walk is bound by its instructions: with 13 of 32 lanes doing useful work
// per instruction (lanes are in different cells, collisions and
// iterations), every instruction of a cell counts.  So its state is scalars that
// stay in registers (arrays indexed by the crossed axis lived in local
// memory), it is inlined, where the medium's constants are operands from the
// constant bank, and a cell's corner differences come ready made in three
// loads instead of nine loads and fourteen additions (512 x 512 x 8 frame of a
// 256^3 grid: 50.2 to 35.1 ms).
struct SvWalk {
    int x, y, z;            // the cell
    float tx, ty, tz;       // distances to its exit planes
};

struct SvSetup {
    V3 invD;                // 1 / direction: the plane distances are multiplications
    SvWalk init;
};

__device__ __forceinline__ float svPlane(float bmin, float width, int cell, bool up) {
    return bmin + width * (cell + (up ? 1 : 0));
}

__device__ __forceinline__ void svSetup(const DevMedium &m, V3 org, V3 dir, float dmin, SvSetup &s) {
    V3 p = mediumLocal(m, org + dmin * dir);
    p = V3{fminf(fmaxf(p.x, 0.0f), 1.0f), fminf(fmaxf(p.y, 0.0f), 1.0f), fminf(fmaxf(p.z, 0.0f), 1.0f)};
    s.invD = V3{1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z};
    s.init.x = min((int)(p.x * (m.svx - 1)), (int)m.svx - 2);
    s.init.y = min((int)(p.y * (m.svy - 1)), (int)m.svy - 2);
    s.init.z = min((int)(p.z * (m.svz - 1)), (int)m.svz - 2);
    s.init.tx = (svPlane(m.bmin[0], m.svWidth[0], s.init.x, dir.x > 0) - org.x) * s.invD.x;
    s.init.ty = (svPlane(m.bmin[1], m.svWidth[1], s.init.y, dir.y > 0) - org.y) * s.invD.y;
    s.init.tz = (svPlane(m.bmin[2], m.svWidth[2], s.init.z, dir.z > 0) - org.z) * s.invD.z;
}

// Cubic in the segment parameter of the trilinear super-voxel majorant
// between entry and exit (plus the cell's maximum difference).
__device__ __forceinline__ void svPolyCoeffs(const DevMedium &m, V3 entry, V3 exit, const SvWalk &w, float c[4]) {
    const float4* cp = reinterpret_cast<const float4*>(
        m.cells + ((m.svx - 1) * (m.svy - 1) * w.z + (m.svx - 1) * w.y + w.x));
    const float4 q0 = __ldg(cp), q1 = __ldg(cp + 1);
    const float maxDiff = __ldg(reinterpret_cast<const float*>(cp + 2));
    const float dxyz = q0.x, dxy = q0.y, dxz = q0.z, dyz = q0.w, dx = q1.x, dy = q1.y, dz = q1.z, d000 = q1.w;
    V3 base = V3{m.bmin[0] + w.x * m.svWidth[0], m.bmin[1] + w.y * m.svWidth[1], m.bmin[2] + w.z * m.svWidth[2]};
    V3 ep = V3{(entry.x - base.x) * m.invSvWidth[0], (entry.y - base.y) * m.invSvWidth[1],
               (entry.z - base.z) * m.invSvWidth[2]};
    V3 op = V3{(exit.x - base.x) * m.invSvWidth[0], (exit.y - base.y) * m.invSvWidth[1],
               (exit.z - base.z) * m.invSvWidth[2]};
    V3 dl = op - ep;
    c[3] = dxyz * dl.x * dl.y * dl.z;
    c[2] = ((ep.z * dl.x * dl.y + ep.y * dl.x * dl.z + ep.x * dl.y * dl.z) * dxyz + dxy * dl.x * dl.y +
            dxz * dl.x * dl.z + dyz * dl.y * dl.z);
    c[1] = ((ep.y * ep.z * dl.x + ep.x * ep.z * dl.y + ep.x * ep.y * dl.z) * dxyz + dx * dl.x + dy * dl.y +
            dz * dl.z + (ep.y * dl.x + ep.x * dl.y) * dxy + (ep.z * dl.x + ep.x * dl.z) * dxz +
            (ep.z * dl.y + ep.y * dl.z) * dyz);
    c[0] = (ep.x * ep.y * ep.z * dxyz + ep.x * ep.y * dxy + ep.x * ep.z * dxz + ep.y * ep.z * dyz + ep.x * dx +
            ep.y * dy + ep.z * dz + d000);
    c[0] += maxDiff;
}

// A tentative collision of the majorant process along [dmin, dmax), the parts
// of traverseSuperVoxels (DensityGridMediumDistribution.cpp:208-367): the
// cells up to the one whose integrated majorant reaches the sampled optical
// depth, then the distance inside that cell.
constexpr int kMaxSvSteps = 4096;
enum SvState : int { kSvWalking = 0, kSvReached = 1, kSvLeft = 2 };

struct SvFlight {
    float sampledOD;
    float exitDist, exitOD;      // of the last cell walked
    float entryDist, entryOD;    // of the cell that reached the sampled depth
    float c[4];                  // its cubic
    int steps;
};

__device__ __forceinline__ void svStart(SvFlight &f, float dmin, float sampledOD) {
    f.sampledOD = sampledOD;
    f.exitDist = dmin;
    f.exitOD = 0.0f;
    f.steps = 0;
}

// One cell.  kSvLeft: the walk leaves the grid, or the segment before its end dmax.
__device__ __forceinline__ int svCell(const DevMedium &m, V3 org, V3 dir, V3 invD, float dmax, float sigma, SvWalk &w,
                                      SvFlight &f) {
    f.entryDist = f.exitDist;
    f.entryOD = f.exitOD;
    const V3 entryP = org + f.entryDist * dir;
    // The axis whose plane comes first; of equal distances the later axis,
    // as the reference's comparison table has it.
    const bool isX = w.tx < w.ty && w.tx < w.tz;
    const bool isY = !(w.tx < w.ty) && w.ty < w.tz;
    f.exitDist = isX ? w.tx : (isY ? w.ty : w.tz);
    const V3 exitP = org + f.exitDist * dir;
    svPolyCoeffs(m, entryP, exitP, w, f.c);
    f.exitOD += (f.exitDist - f.entryDist) * sigma * (f.c[0] + f.c[1] * 0.5f + f.c[2] * kThird + f.c[3] * 0.25f);
    if (f.exitOD >= f.sampledOD) return kSvReached;
    // one cell along the axis; out of the grid on either side ends the walk
    const float da = isX ? dir.x : (isY ? dir.y : dir.z);
    const bool up = da > 0;
    const int cell = (isX ? w.x : (isY ? w.y : w.z)) + (up ? 1 : -1);
    const int outside = up ? (int)(isX ? m.svx : (isY ? m.svy : m.svz)) - 1 : -1;
    const float bmin = isX ? m.bmin[0] : (isY ? m.bmin[1] : m.bmin[2]);
    const float width = isX ? m.svWidth[0] : (isY ? m.svWidth[1] : m.svWidth[2]);
    const float oa = isX ? org.x : (isY ? org.y : org.z);
    const float inv = isX ? invD.x : (isY ? invD.y : invD.z);
    const bool left = cell == outside || f.exitDist >= dmax || ++f.steps > kMaxSvSteps;
    const float t = (svPlane(bmin, width, cell, up) - oa) * inv;
    if (isX) { w.x = cell; w.tx = left ? w.tx : t; }
    else if (isY) { w.y = cell; w.ty = left ? w.ty : t; }
    else { w.z = cell; w.tz = left ? w.tz : t; }
    return left ? kSvLeft : kSvWalking;
}

// Regula falsi on the integrated majorant of the cell that reached the
// sampled depth.  Returns false (and *dist = dmax) past the segment's end.
__device__ __forceinline__ bool svDistance(const SvFlight &f, float dmax, float sigma, float* dist, float* majorant) {
    const float* c = f.c;
    float pLow = 0.0f, pHigh = 1.0f, odLow = f.entryOD, odHigh = f.exitOD;
    float prev = -__int_as_float(0x7f800000), cur = pHigh;
    int iters = 0;
    while (fabsf(cur - prev) >= 1e-3f * fabsf(cur) && iters < 100) {
        prev = cur;
        cur = pLow + (pHigh - pLow) * __fdividef(f.sampledOD - odLow, odHigh - odLow);
        float temp = sigma * (c[0] * cur + c[1] * cur * cur * 0.5f + c[2] * cur * cur * cur * kThird +
                              c[3] * cur * cur * cur * cur * 0.25f);
        float od = f.entryOD + (f.exitDist - f.entryDist) * temp;
        ++iters;
        if (od < f.sampledOD) { pLow = cur; odLow = od; }
        else if (od > f.sampledOD) { pHigh = cur; odHigh = od; }
        else break;
    }
    *dist = f.entryDist + (f.exitDist - f.entryDist) * cur;
    if (*dist >= dmax) {
        *dist = dmax;
        *majorant = __int_as_float(0x7fc00000);
        return false;
    }
    *majorant = sigma * (c[0] + c[1] * cur + c[2] * cur * cur + c[3] * cur * cur * cur);
    return true;
}

// The whole of it for one thread.  Returns false (and *dist = dmax) when the
// walk leaves the segment.
__device__ __forceinline__ bool svTraverse(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax, float u,
                                           float sigma, const SvSetup &s, SvWalk &w, float* dist, float* majorant) {
    const float sampledOD = -logf(1 - u);
    if (sampledOD == 0.0f) {
        V3 q = org + (*dist) * dir;
        *majorant = sigma * mediumCoarseDensity(m, mediumLocal(m, q));
        return true;
    }
    SvFlight f;
    svStart(f, dmin, sampledOD);
    int state;
    do state = svCell(m, org, dir, s.invD, dmax, sigma, w, f);
    while (state == kSvWalking);
    if (state == kSvLeft) {
        *dist = dmax;
        *majorant = __int_as_float(0x7fc00000);
        return false;
    }
    return svDistance(f, dmax, sigma, dist, majorant);
}

// DensityGridMediumDistribution::interact (:402-575): delta tracking at the
// selected wavelength; spectral throughput for the others by the ratio
// estimator.  Returns true on a real collision at *tHit (param = normalised
// position).  thr receives the medium throughput (already divided by the
// extinction coefficient at the collision).
template <class R>
__device__ __noinline__ bool mediumInteractSegment(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                                   const Spec &sigmaE, int sel, bool wlSelected, R &rng,
                                                   float* tHit, V3* param, Spec &thr) {
    SvSetup s;
    svSetup(m, org, dir, dmin, s);
    SvWalk w = s.init;
    bool hit = false;
    float extAt = 0.0f;
    float sd = dmin;
    const float sigSel = specAt(sigmaE, sel);
    while (sd < dmax) {
        float maj;
        bool tent = svTraverse(m, org, dir, sd, dmax, rng.next(), sigSel, s, w, &sd, &maj);
        if (!tent) { hit = false; break; }
        V3 q = org + sd * dir;
        V3 pr = mediumLocal(m, q);
        float ext = sigSel * mediumDensity(m, pr);
        float prob = ext / maj;
        if (rng.next() < prob) {
            hit = true;
            *tHit = sd;
            *param = pr;
            extAt = ext;
            break;
        }
    }
    if (wlSelected) {
#pragma unroll
        for (int k = 0; k < kNumLambda; ++k) thr.v[k] = (k == sel) ? 1.0f : 0.0f;
    } else {
        const float hitDist = fminf(sd, dmax);
        sd = dmin;
        w = s.init;
        // The walk state is shared across the wavelengths, so only the first
        // wavelength other than the selected one takes steps (the reference's
        // loop at DensityGridMediumDistribution.cpp:487-510 never resets it).
        const int wl = sel == 0 ? 1 : 0;
        const float sigWl = wl == 0 ? sigmaE.v[0] : sigmaE.v[1];
        float mc = 1.0f;
        while (sd < hitDist) {
            float maj;
            bool tent = svTraverse(m, org, dir, sd, hitDist, rng.next(), sigWl, s, w, &sd, &maj);
            if (tent) {
                V3 q = org + sd * dir;
                float dens = mediumDensity(m, mediumLocal(m, q));
                float prob = (sigWl * dens - sigSel * dens) / maj;
                if (maj != 0.0f) mc *= (1.0f - prob);
            }
        }
#pragma unroll
        for (int k = 0; k < kNumLambda; ++k) thr.v[k] = k == wl ? mc : 1.0f;
    }
    if (hit) {
        float r = 1.0f / extAt;
#pragma unroll
        for (int k = 0; k < kNumLambda; ++k) thr.v[k] *= r;
    }
    return hit;
}

// Ratio-tracking estimate of one wavelength's transmittance over [dmin, dmax)
// inside the medium, with Russian roulette below 0.1
// (DensityGridMediumDistribution.cpp:618-651); s is the DDA set-up at dmin.
template <class R>
__device__ __forceinline__ float ratioTrackSegment(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                                   const SvSetup &s, float sig, R &rng) {
    float t = 1.0f;
    SvWalk w = s.init;
    float sd = dmin;
    while (sd < dmax) {
        float maj;
        bool tent = svTraverse(m, org, dir, sd, dmax, rng.next(), sig, s, w, &sd, &maj);
        if (tent) {
            float ext = sig * mediumDensity(m, mediumLocal(m, org + sd * dir));
            float prob = ext / maj;
            if (maj != 0.0f) t *= (1.0f - prob);
            if (t < 0.1f) {
                if (rng.next() < t) t = 1.0f;
                else return 0.0f;
            }
        }
    }
    return t;
}

// Spectral transmittance of one segment inside the medium
// (DensityGridMediumDistribution::evaluateTransmittance, :577-744): every
// wavelength, or only the selected one once a wavelength is selected.
template <class R>
__device__ __noinline__ void mediumTransmittanceSegment(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                                        const Spec &sigmaE, int sel, bool wlSelected, R &rng,
                                                        Spec &T) {
    SvSetup s;
    svSetup(m, org, dir, dmin, s);
    T = specConst(0.0f);
    for (int wl = 0; wl < kNumLambda; ++wl) {
        if (wlSelected && wl != sel) continue;
        const float t = ratioTrackSegment(m, org, dir, dmin, dmax, s, specAt(sigmaE, wl), rng);
#pragma unroll
        for (int k = 0; k < kNumLambda; ++k)
            if (k == wl) T.v[k] = t;
    }
}

// MediumObjectAggregate::interact for one medium (medium_object.cpp:287-348):
// walks boundary crossings of the medium box within [dmin, dmax).
template <class R>
__device__ __forceinline__ bool mediumInteract(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                               const Spec &sigmaE, int sel, bool wlSelected, R &rng, float* tHit,
                                               V3* param, Spec &thr) {
    thr = specConst(1.0f);
    float rmin = dmin;
    bool inside = mediumContains(m, org + rmin * dir);
    for (int guard = 0; guard < 8; ++guard) {
        float dist;
        bool enter;
        bool nextInside = false;
        float distNext = __int_as_float(0x7f800000);
        if (mediumIntersectBoundary(m, org, dir, rmin, dmax, &dist, &enter) && dist < distNext) {
            distNext = dist;
            nextInside = enter;
        }
        if (inside && nextInside) inside = false;
        distNext = fminf(distNext, dmax);
        if (isinf(distNext)) return false;
        if (inside) {
            Spec t;
            bool hit = mediumInteractSegment(m, org, dir, rmin, distNext, sigmaE, sel, wlSelected, rng, tHit, param, t);
#pragma unroll
            for (int k = 0; k < kNumLambda; ++k) thr.v[k] *= t.v[k];
            if (hit) return true;
        }
        if (distNext == dmax) return false;
        rmin = distNext * (1.0f + kRayEpsilon);
        inside = nextInside;
    }
    return false;
}

// MediumObjectAggregate::evaluateTransmittance for one medium (:350-402).
template <class R>
__device__ __forceinline__ void mediumTransmittance(const DevMedium &m, V3 org, V3 dir, float dmin, float dmax,
                                                    const Spec &sigmaE, int sel, bool wlSelected, R &rng, Spec &T) {
    T = specConst(1.0f);
    float rmin = dmin;
    bool inside = mediumContains(m, org + rmin * dir);
    for (int guard = 0; guard < 8; ++guard) {
        float dist;
        bool enter;
        bool nextInside = false;
        float distNext = __int_as_float(0x7f800000);
        if (mediumIntersectBoundary(m, org, dir, rmin, dmax, &dist, &enter) && dist < distNext) {
            distNext = dist;
            nextInside = enter;
        }
        if (inside && nextInside) inside = false;
        distNext = fminf(distNext, dmax);
        if (isinf(distNext)) return;
        if (inside) {
            Spec t;
            mediumTransmittanceSegment(m, org, dir, rmin, distNext, sigmaE, sel, wlSelected, rng, t);
#pragma unroll
            for (int k = 0; k < kNumLambda; ++k) T.v[k] *= t.v[k];
        }
        if (distNext == dmax) return;
        rmin = distNext * (1.0f + kRayEpsilon);
        inside = nextInside;
    }
}

// One wavelength of mediumTransmittance, for one lane per (ray, wavelength):
// the same boundary crossings and per-segment ratio tracking, its state kept
// between the steps of trRun.  `evaluate` false (a wavelength other than the
// selected one) gives 0 once the ray crosses the medium and 1 otherwise, as
// the spectral version does.
struct TrWalk {
    V3 org, dir;
    float dmax, sig;
    uint64_t key;       // of the walk's random numbers
    uint32_t counter;
    float T;            // product of the finished segments
    float t;            // the current segment's ratio-tracking estimate
    float rmin, segEnd, sd;
    int guard;
    bool inside, nextInside, evaluate;
    SvSetup s;
    SvWalk w;
};

// Runs the boundary loop until a segment inside the medium is ready to walk
// (true) or the estimate q.T is final (false).
__device__ __forceinline__ bool trAdvance(const DevMedium &m, TrWalk &q) {
    for (; q.guard < 8; ++q.guard) {
        float dist;
        bool enter;
        q.nextInside = false;
        float distNext = __int_as_float(0x7f800000);
        if (mediumIntersectBoundary(m, q.org, q.dir, q.rmin, q.dmax, &dist, &enter) && dist < distNext) {
            distNext = dist;
            q.nextInside = enter;
        }
        if (q.inside && q.nextInside) q.inside = false;
        distNext = fminf(distNext, q.dmax);
        if (isinf(distNext)) return false;
        q.segEnd = distNext;
        if (q.inside) {
            if (!q.evaluate) {
                q.T = 0.0f;
                return false;
            }
            svSetup(m, q.org, q.dir, q.rmin, q.s);
            q.w = q.s.init;
            q.t = 1.0f;
            q.sd = q.rmin;
            if (q.sd < q.segEnd) return true;
            q.T *= q.t;      // an empty segment estimates 1
        }
        if (q.segEnd == q.dmax) return false;
        q.rmin = q.segEnd * (1.0f + kRayEpsilon);
        q.inside = q.nextInside;
    }
    return false;
}

__device__ __forceinline__ bool trBegin(const DevMedium &m, TrWalk &q, V3 org, V3 dir, float dmin, float dmax,
                                        float sig, bool evaluate, uint64_t key, uint32_t counter) {
    q.org = org;
    q.dir = dir;
    q.dmax = dmax;
    q.sig = sig;
    q.evaluate = evaluate;
    q.key = key;
    q.counter = counter;
    q.T = 1.0f;
    q.rmin = dmin;
    q.guard = 0;
    q.inside = mediumContains(m, org + dmin * dir);
    return trAdvance(m, q);
}

// After a tentative collision at q.sd with majorant maj (tent), or the end of
// the segment: ratioTrackSegment's loop body.  Returns true while the walk
// goes on; q.T is final otherwise.
__device__ __forceinline__ bool trCollide(const DevMedium &m, TrWalk &q, bool tent, float maj) {
    bool segDone = !(q.sd < q.segEnd);
    if (tent) {
        float ext = q.sig * mediumDensity(m, mediumLocal(m, q.org + q.sd * q.dir));
        float prob = ext / maj;
        if (maj != 0.0f) q.t *= (1.0f - prob);
        if (q.t < 0.1f) {
            if (uniformFloat(q.key, q.counter++) < q.t) {
                q.t = 1.0f;
            } else {
                q.t = 0.0f;
                segDone = true;
            }
        }
    }
    if (!segDone) return true;
    q.T *= q.t;
    if (q.T == 0.0f) return false;
    if (q.segEnd == q.dmax) return false;
    q.rmin = q.segEnd * (1.0f + kRayEpsilon);
    q.inside = q.nextInside;
    ++q.guard;
    return trAdvance(m, q);
}

// Hands out work items [0, n) to the lanes of a warp that ask for one, in
// chunks of kTrChunk taken from a global counter (one atomic per chunk).
// All 32 lanes call it together; the chunk range is the same in every lane.
constexpr uint32_t kTrChunk = 64;

__device__ __forceinline__ uint32_t trTake(bool need, uint32_t* take, uint32_t &poolNext, uint32_t &poolEnd) {
    const unsigned mask = __ballot_sync(0xffffffffu, need);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t k = __popc(mask), rank = __popc(mask & ((1u << lane) - 1));
    uint32_t item = poolNext + rank;
    const uint32_t avail = poolEnd - poolNext;
    if (k > avail) {
        uint32_t c = 0;
        if (lane == 0) c = atomicAdd(take, kTrChunk);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (rank >= avail) item = c + (rank - avail);
        poolNext = c + (k - avail);
        poolEnd = c + kTrChunk;
    } else {
        poolNext += k;
    }
    return item;
}

// The walks of work items [0, n) by all lanes of the calling warps.  begin(item,
// q) starts an item's walk (false: it had none, or its result is dealt with);
// end(item, q) takes the final estimate q.T.
//
// Bound by instructions, and so by how many lanes do useful work in each: a
// walk alternates between cells (one to eight per collision), the distance
// inside the last one (three to seven iterations), the collision and a new
// draw, and a lane that ran each to its end had the others wait for the
// longest (12.7 of 32 lanes at work).  So the warp advances cell by cell until
// fewer than a quarter of its live lanes are still between cells, then deals
// with the collisions and segment ends together while the others keep their
// place (16.7 lanes at work with a half), and fills idle lanes (a start costs
// six divisions) a quarter warp at a time.  512 x 512 x 8 frame of a 256^3
// grid: 35.1 ms with every lane run to its collision, 33.1 with
// the line at a half of the live lanes, 32.7 at a quarter, 34.1 at
// an eighth; refills at 4 or 16 idle lanes 32.8 and 33.4.
#ifndef SLRGPU_TR_REFILL
#define SLRGPU_TR_REFILL 8
#endif
#ifndef SLRGPU_TR_WAIT
#define SLRGPU_TR_WAIT 4
#endif
template <class Begin, class End>
__device__ __forceinline__ void trRun(const DevMedium &m, uint32_t n, uint32_t* take, Begin begin, End end) {
    constexpr unsigned kAll = 0xffffffffu;
    enum { kIdle = 3, kDraw = 4, kCollide = 5 };   // besides the SvState values
    uint32_t poolNext = 0, poolEnd = 0, item = 0;
    bool exhausted = false;
    int state = kIdle;
    TrWalk q;
    SvFlight f;
    float maj = 0.0f;
    for (;;) {
        for (;;) {
            const bool need = state == kIdle && !exhausted;
            const unsigned idle = __ballot_sync(kAll, need);
            if (idle == 0) break;
            if (__popc(idle) < SLRGPU_TR_REFILL && __any_sync(kAll, state != kIdle)) break;
            const uint32_t it = trTake(need, take, poolNext, poolEnd);
            if (!need) continue;
            item = it;
            if (it >= n) exhausted = true;
            else if (begin(it, q)) state = kDraw;
        }
        const unsigned live = (unsigned)__popc(__ballot_sync(kAll, state != kIdle));
        if (live == 0) return;
        if (state == kDraw) {
            const float sampledOD = -logf(1 - uniformFloat(q.key, q.counter++));
            if (sampledOD == 0.0f) {
                maj = q.sig * mediumCoarseDensity(m, mediumLocal(m, q.org + q.sd * q.dir));
                state = kCollide;
            } else {
                svStart(f, q.sd, sampledOD);
                state = kSvWalking;
            }
        }
        for (;;) {
            const unsigned walking = (unsigned)__popc(__ballot_sync(kAll, state == kSvWalking));
            if (walking == 0 || SLRGPU_TR_WAIT * walking < live) break;
            if (state == kSvWalking) state = svCell(m, q.org, q.dir, q.s.invD, q.segEnd, q.sig, q.w, f);
        }
        if (state == kSvReached) state = svDistance(f, q.segEnd, q.sig, &q.sd, &maj) ? (int)kCollide : (int)kSvLeft;
        else if (state == kSvLeft) q.sd = q.segEnd;
        if (state == kCollide || state == kSvLeft) {
            if (trCollide(m, q, state == kCollide, maj)) {
                state = kDraw;
            } else {
                end(item, q);
                state = kIdle;
            }
        }
    }
}

// Henyey-Greenstein phase function (PhaseFunction/basic_phase_functions.cpp:36-65).
__device__ __forceinline__ float hgValue(float g, float cosTheta) {
    return (1 - g * g) / (4 * kPiF * powf(1 + g * g - 2 * g * cosTheta, 1.5f));
}

__device__ __forceinline__ V3 hgSample(float g, float u0, float u1, float* pdf) {
    float sq = (1 - g * g) / (1 - g + 2 * g * u1);
    float cosTheta = fminf(fmaxf(0.5f / g * (1 + g * g - sq * sq), -1.0f), 1.0f);
    float phi = 2 * kPiF * u0;
    *pdf = hgValue(g, cosTheta);
    float sinTheta = sqrtf(1 - cosTheta * cosTheta);
    float sp, cp;
    sincosf(phi, &sp, &cp);
    return V3{cp * sinTheta, sp * sinTheta, cosTheta};
}

// ReferenceFrame(z) with Duff et al.'s orthonormal basis (Vector3D.h:59-66).
__device__ __forceinline__ Frame frameFromZ(V3 z) {
    float sign = z.z >= 0.0f ? 1.0f : -1.0f;
    const float a = -1.0f / (sign + z.z);
    const float b = z.x * z.y * a;
    V3 x = V3{1.0f + sign * z.x * z.x * a, sign * b, -sign * z.x};
    V3 y = V3{b, sign + z.y * z.y * a, -z.y};
    return Frame{x, y, z};
}

}  // namespace slrgpu
