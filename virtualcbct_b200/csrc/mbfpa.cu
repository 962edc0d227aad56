// mbfpa.cu -- material-based polychromatic forward projection (MBFPA) on sm_100a.
//
// Reference: Release_CBCT_Projection_CM/reprojectionOnGPU.cu (reprojectionKernel,
// :56-690, launched once per energy bin from :1004-1056).  This file keeps its
// per-ray semantics -- the Siddon-style march with its discrete rules -- and
// changes how the work maps to the GPU:
//
//  * one launch marches every ray once and accumulates the six per-element
//    path integrals L_k; the spectral sum  leng * sum_E pdf_E exp(-sum_k
//    mu_k(E) L_k / xfactor)  is formed in the same kernel (the reference
//    re-marches every ray for each of ~100 bins and copies the whole stack to
//    the host after each);
//  * a warp is 32 consecutive detector rows of one column: those rays share
//    their xy trajectory, so trip counts and x/y plane crossings are
//    warp-uniform and only z crossings diverge;
//  * where several of those rays lie in one slice, their sums over a chunk of
//    intervals are made once per slice in shared memory (column march);
//  * the volume is re-laid out once into z-fastest voxel records, 16 bytes of
//    uint16 or 32 of floats (all elements of a voxel in one vector load); the
//    warp's loads at a step fall in one contiguous run of a z column;
//  * FP64 is used only for the per-ray source/detector geometry, the
//    entry/exit and loop-bound computation, and the parametric positions
//    (Siddon alphas) of plane crossings.  The march itself is FP32, with
//    voxel cells carried as integers plus a small fractional offset so that no
//    FP32 value has to resolve a large coordinate near a plane.
//
// Also here: the band footprints of the host-to-host pipelined projection,
// the batch kernels (persistent work queue, flat tile list), the adjoint
// (per-ray spectral derivative, then the same segments scattered into
// z-fastest planes of element groups, summed per slice first where rays share
// one, optionally restricted to a strip of volume rows), and the volume /
// gradient re-layout kernels.
#include "internal.h"
#include "noise.cuh"

#include <cfloat>
#include <climits>
#include <type_traits>

namespace vcbct {

size_t packed_u16_bytes(int N, int Z) { return (size_t)N * N * Z * sizeof(uint4); }
size_t packed_f32_bytes(int N, int Z) { return (size_t)N * N * Z * 2 * sizeof(float4); }

namespace {

// ---------------------------------------------------------------- FP64 ops --
// Explicitly rounded double operations: nvcc may not contract these into
// FMAs, so the setup reproduces the reference's double arithmetic bitwise.
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// (a - a0)/(a1 - a0)*(b1 - b0) + b0, the reference's line evaluation (:159).
__device__ __forceinline__ double line_at(double a, double a0, double a1, double b0, double b1)
{
    return dadd(dmul(ddiv(dsub(a, a0), dsub(a1, a0)), dsub(b1, b0)), b0);
}

// (int) cast of a double made total (non-finite / out of range -> INT_MIN).
__device__ __forceinline__ int d2i(double v)
{
    if (!(v > -2147483648.0 && v < 2147483647.0)) return INT_MIN;
    return __double2int_rz(v);
}

constexpr float kInf = 3.0e38f;

// One axis of the march: value(t) = I + F + slope * (t - ta), in voxel (or
// slice) units.  I is an integer cell base, F a small fraction.
struct Axis {
    int I;
    float F;
    float slope;
    float ta;
};

__device__ __forceinline__ float axis_frac(const Axis& a, float t)
{
    return fmaf(a.slope, t - a.ta, a.F);
}

// Everything the FP32 march needs about one ray, produced by ray_setup().
struct RayPlan {
    int active;      // emits at least one segment
    int d;           // dominant axis (0: x, 1: y)
    int pha;         // +1 / -1 along the dominant axis
    int kstar;       // last iteration index (iterations 0..kstar)
    int klo, khi;    // iterations k >= 1 that can contribute (inclusive)
    int first_idx;   // packed voxel of the first segment, or -1
    float first_len; // its length [cm]
    float Lt;        // cm per unit of t
    float leng;      // cos^3 factor (reprojectionOnGPU.cu:141-150)
    double D0;       // dominant coordinate / s at t = 0
    double O0, O1;   // other in-plane coordinate / s:  O0 + O1 t
    double Z0, Z1;   // z / step:                        Z0 + Z1 t
    double invO1, invZ1;  // 1 / O1, 1 / Z1 (0 when the slope is 0)
    double tc0, tc1; // chord of the cylindrical mask in t
};

// Per-ray FP64 setup: reprojectionOnGPU.cu:128-212, mirrored operation for
// operation.  Rays that hit the xy square fewer than twice are defined to miss
// (the reference reads uninitialised entries there).  Written with scalars and
// selects instead of small arrays indexed by the ray's axes, and inlined, so
// the plan stays in registers (no per-ray stack traffic).
__device__ __forceinline__ void ray_setup(const ProjParams& P, const ViewGeom& vg, int j, int jj, RayPlan& R)
{
    const double s = P.s, step = P.step;
    const int nxm = (int)(P.N * 0.5), nym = (int)(P.N * 0.5), nzm = (int)(P.Z * 0.5);
    const double S0 = dadd(dmul(-P.sad, vg.sn), P.xr);
    const double S1 = dadd(dmul(P.sad, vg.cs), P.yr);
    const double S2 = P.zr;
    const double bin = ddiv(P.dpn, (double)P.H);
    const double P2 = dadd(dmul(dmul(-dadd(vg.yc, (double)j), P.piso), bin), ddiv(dmul(P.zr, P.piso), P.pdet));
    const double pr = dmul(dmul(P.piso, dadd(vg.xc, (double)jj)), bin);
    const double P0 = dadd(dmul(pr, vg.cs), ddiv(dmul(P.xr, P.piso), P.pdet));
    const double P1 = dadd(dmul(pr, vg.sn), ddiv(dmul(P.yr, P.piso), P.pdet));
    {
        const double d2 = dmul(P.sad, P.sad);
        double l = ddiv(d2, dadd(d2, dadd(dmul(pr, pr), dmul(P2, P2))));
        R.leng = (float)dmul(l, __dsqrt_rn(l));
    }
    R.active = 0;
    R.klo = INT_MAX;
    R.khi = -1;
    R.first_idx = -1;
    R.first_len = 0.0f;

    // entry / exit against the four side planes (:154-183); only the first
    // two hits are used, so only they are kept
    const double hx = dmul((double)nxm, s), hy = dmul((double)nym, s);
    double hx0 = 0.0, hy0 = 0.0, hz0 = 0.0, hx1 = 0.0, hy1 = 0.0, hz1 = 0.0;
    int m = 0;
    auto hit = [&](double x, double y, double z) {
        if (m == 0) { hx0 = x; hy0 = y; hz0 = z; }
        else if (m == 1) { hx1 = x; hy1 = y; hz1 = z; }
        m++;
    };
    if (fabs(line_at(hy, S1, P1, S0, P0)) < hx) hit(line_at(hy, S1, P1, S0, P0), hy, line_at(hy, S1, P1, S2, P2));
    if (fabs(line_at(-hy, S1, P1, S0, P0)) < hx) hit(line_at(-hy, S1, P1, S0, P0), -hy, line_at(-hy, S1, P1, S2, P2));
    if (fabs(line_at(hx, S0, P0, S1, P1)) < hy) hit(hx, line_at(hx, S0, P0, S1, P1), line_at(hx, S0, P0, S2, P2));
    if (fabs(line_at(-hx, S0, P0, S1, P1)) < hy) hit(-hx, line_at(-hx, S0, P0, S1, P1), line_at(-hx, S0, P0, S2, P2));
    if (m < 2) return;

    // entry I = the hit nearer the source, exit F = the other
    double I0, I1, I2, F0, F1;
    {
        const double e0 = dadd(dadd(dmul(dsub(hx0, S0), dsub(hx0, S0)), dmul(dsub(hy0, S1), dsub(hy0, S1))),
                               dmul(dsub(hz0, S2), dsub(hz0, S2)));
        const double e1 = dadd(dadd(dmul(dsub(hx1, S0), dsub(hx1, S0)), dmul(dsub(hy1, S1), dsub(hy1, S1))),
                               dmul(dsub(hz1, S2), dsub(hz1, S2)));
        const bool f0 = e0 < e1;
        I0 = f0 ? hx0 : hx1; I1 = f0 ? hy0 : hy1; I2 = f0 ? hz0 : hz1;
        F0 = f0 ? hx1 : hx0; F1 = f0 ? hy1 : hy0;
    }
    // dominant axis, GPU twin rule (:198); _d / _o name the dominant and the
    // other in-plane axis
    const int d = (fabs(dsub(I0, F0)) > fabs(dsub(I1, F1))) ? 0 : 1;
    const double Id = d ? I1 : I0, Fd = d ? F1 : F0;
    const double Sd = d ? S1 : S0, So = d ? S0 : S1;
    const double Pd = d ? P1 : P0, Po = d ? P0 : P1;
    const double dF = dsub(Fd, Id);
    const double pha = ddiv(dF, fabs(dsub(Id, Fd)));
    if (!(pha == 1.0 || pha == -1.0)) return;
    int ain;
    if ((Id < 0 && dF < 0) || (Id > 0 && dF > 0))
        ain = d2i(dadd((double)d2i(Id), ddiv(dF, fabs(dF))));
    else
        ain = d2i(Id);
    if (ain == INT_MIN) return;

    const double h = hx;  // hx == hy (both from reconSize)
    auto inb = [&](double k) {
        double a = dadd((double)ain, dmul(dmul(pha, k), s));
        double ov = line_at(a, Sd, Pd, So, Po);
        return a <= h && a >= -h && ov <= h && ov >= -h;
    };
    if (!inb(0.0)) return;

    // first iteration whose step point leaves the box; the loop of the
    // reference (:212) executes it and stops.
    const double go = ddiv(dsub(Po, So), dsub(Pd, Sd));
    const double gz = ddiv(dsub(P2, S2), dsub(Pd, Sd));
    const double o0 = line_at((double)ain, Sd, Pd, So, Po);
    const double z0 = line_at((double)ain, Sd, Pd, S2, P2);
    double kd = floor((h - pha * ain) / s) + 1.0;
    double ko = 1e30;
    const double vo = go * pha * s;
    if (vo > 0) ko = floor((h - o0) / vo) + 1.0;
    else if (vo < 0) ko = floor((-h - o0) / vo) + 1.0;
    double ke = fmin(kd, ko);
    const int kcap = 4 * (P.N + 4) + (int)(8.0 / s) + 64;
    if (!(ke >= 1.0)) ke = 1.0;
    if (ke > kcap) ke = kcap;
    int ks = (int)ke;
    while (ks > 1 && !inb((double)(ks - 1))) ks--;
    int guard = 0;
    while (inb((double)ks) && guard < kcap) { ks++; guard++; }
    R.kstar = ks;

    R.d = d;
    R.pha = (int)pha;
    R.D0 = (double)ain / s;
    R.O0 = o0 / s;
    R.O1 = go * pha;
    R.Z0 = z0 / step;
    R.Z1 = gz * pha * s / step;
    R.Lt = (float)(s * sqrt(1.0 + go * go + gz * gz));
    R.invO1 = (R.O1 != 0.0) ? 1.0 / R.O1 : 0.0;
    R.invZ1 = (R.Z1 != 0.0) ? 1.0 / R.Z1 : 0.0;
    R.tc0 = 1.0;
    R.tc1 = 0.0;
    R.active = 1;

    // Iteration 0 emits one unsplit segment from the entry point to the first
    // step point (:405-427 with ik == 0).  It can span many voxels and its
    // midpoint often lies exactly on a voxel plane (entry through a face), so
    // its voxel, length and mask are evaluated in FP64 exactly as the
    // reference does.
    {
        const double b10 = d ? o0 : (double)ain;
        const double b11 = d ? (double)ain : o0;
        const double b12 = z0;
        const double rr = __dsqrt_rn(dadd(dadd(dmul(dsub(I0, b10), dsub(I0, b10)),
                                               dmul(dsub(I1, b11), dsub(I1, b11))),
                                          dmul(dsub(I2, b12), dsub(I2, b12))));
        const int xmc = d2i(dadd(ddiv(dmul(dadd(I0, b10), 0.5), s), (double)nxm));
        const int ymc = d2i(dadd(ddiv(dmul(dsub(-I1, b11), 0.5), s), (double)nym));
        const int zmc = d2i(dadd(ddiv(dmul(dsub(-I2, b12), 0.5), step), (double)nzm));
        if (xmc >= 0 && ymc >= 0 && zmc >= 0 && xmc <= P.N - 1 && ymc <= P.N - 1 && zmc <= P.Z - 1) {
            const double r = dmul(__dsqrt_rn(dadd(dmul(dadd(I0, b10), dadd(I0, b10)),
                                                  dmul(dsub(-I1, b11), dsub(-I1, b11)))), 0.5);
            if (!(r >= dmul(dmul((double)P.N, 0.5), s))) {
                R.first_idx = (ymc * P.N + xmc) * P.Z + zmc;
                R.first_len = (float)rr;
            }
        }
    }

    // iterations whose segments can pass the cylinder mask and the z bounds
    const double Rv = P.N * 0.5;
    double A = 1.0 + R.O1 * R.O1;
    double B = 2.0 * (R.D0 * pha + R.O0 * R.O1);
    double C = R.D0 * R.D0 + R.O0 * R.O0 - Rv * Rv;
    double disc = B * B - 4.0 * A * C;
    if (!(disc > 0.0)) return;
    double sq = sqrt(disc);
    double tl = (-B - sq) / (2.0 * A), th = (-B + sq) / (2.0 * A);
    R.tc0 = tl;
    R.tc1 = th;
    const double zlo = (double)(nzm - P.Z), zhi = (double)(nzm + 1);  // (int) of zmc in [0, Z-1]
    if (R.Z1 > 0) {
        tl = fmax(tl, (zlo - R.Z0) / R.Z1);
        th = fmin(th, (zhi - R.Z0) / R.Z1);
    } else if (R.Z1 < 0) {
        tl = fmax(tl, (zhi - R.Z0) / R.Z1);
        th = fmin(th, (zlo - R.Z0) / R.Z1);
    } else if (!(R.Z0 > zlo && R.Z0 < zhi)) {
        return;
    }
    if (!(th > tl)) return;
    // iteration k >= 1 covers t in [k-1, k]; one step of margin each side
    int klo = (int)fmax(1.0, floor(tl) - 1.0);
    int khi = (int)fmin((double)ks, floor(th) + 2.0);
    if (khi < klo) return;
    R.klo = klo;
    R.khi = khi;
}

// Map a cell index to the reference's (int)-truncated voxel index: the value
// lies in (q, q+1); q >= 0 -> q, q == -1 -> 0 (truncation toward zero), else
// out of range.  Returns -1 when out of [0, size).
__device__ __forceinline__ int trunc_index(int q, int size)
{
    return ((unsigned)(q + 1) <= (unsigned)size) ? max(q, 0) : -1;
}

// Slice index of a ray with Z1 == 0 (it stays in the plane z = Z0 * step;
// with z_reg = 0 the central detector row does).  The reference's rule
// (int)(nzm - z/step) differs from the cell rule when Z0 is an integer (the
// midpoints then lie exactly on a slice boundary), so it is applied as is.
__device__ __forceinline__ int flat_z_index(const ProjParams& P, double Z0)
{
    const double q = (double)(int)(P.Z * 0.5) - Z0;
    return (q > -1.0 && q < (double)P.Z) ? (int)q : -1;
}

// Anchor of an axis at parameter t (FP64 value v = c0 + c1 t).
__device__ __forceinline__ Axis make_axis(double c0, double c1, double t)
{
    double v = c0 + c1 * t;
    double fl = floor(v);
    Axis a;
    a.I = (int)fl;
    a.F = (float)(v - fl);
    a.slope = (float)c1;
    a.ta = (float)t;
    return a;
}

// Parameter of the crossing of plane `m` (FP64 Siddon alpha, as float).
__device__ __forceinline__ float cross_t(double c0, double inv1, int m)
{
    return (float)(((double)m - c0) * inv1);
}

// The FP32 march of iterations k in [Klo, Khi] (k >= 1) of one ray
// (reprojectionOnGPU.cu:200-429 and its y-dominant mirror :441-666).
// `visit(idx, len)` is called with the packed voxel index of every segment
// that passes the voxel-bounds test and the cylinder mask.
template <class Visit>
__device__ __forceinline__ void march(const ProjParams& P, const RayPlan& R, int Klo, int Khi,
                                      Visit& visit)
{
    const int nxm = (int)(P.N * 0.5), nym = (int)(P.N * 0.5), nzm = (int)(P.Z * 0.5);
    const float R2 = (float)(P.N * 0.5) * (float)(P.N * 0.5);
    const int d = R.d;
    const float fpha = (float)R.pha;
    const double Dfl = floor(R.D0);
    const int Id0 = (int)Dfl;
    const float Fd = (float)(R.D0 - Dfl);

    // o / z crossing bookkeeping (FP64 alphas)
    const int diro = (R.O1 > 0) ? 1 : ((R.O1 < 0) ? -1 : 0);
    const int dirz = (R.Z1 > 0) ? 1 : ((R.Z1 < 0) ? -1 : 0);
    const double invO1 = diro ? 1.0 / R.O1 : 0.0;
    const double invZ1 = dirz ? 1.0 / R.Z1 : 0.0;

    const int ks = Klo;
    const double t0s = (double)(ks - 1);
    Axis ao = make_axis(R.O0, R.O1, t0s);
    Axis az = make_axis(R.Z0, R.Z1, t0s);
    int mo = 0, mz = 0;
    float to_next = kInf, tz_next = kInf;
    if (diro) {
        double v = R.O0 + R.O1 * t0s;
        mo = (diro > 0) ? (int)floor(v) + 1 : (int)ceil(v) - 1;
        to_next = cross_t(R.O0, invO1, mo);
    }
    if (dirz) {
        double v = R.Z0 + R.Z1 * t0s;
        mz = (dirz > 0) ? (int)floor(v) + 1 : (int)ceil(v) - 1;
        if (mz == 0) mz += dirz;  // z = 0 is never a split plane (:237-238)
        tz_next = cross_t(R.Z0, invZ1, mz);
    }

    const int izflat = dirz ? -1 : flat_z_index(P, R.Z0);

    // One segment [ta, tb] within the step whose start is t = tbase, where the
    // dominant cell base is Idk.
    auto segment = [&](float ta, float tb, float tbase, int Idk) {
        const float tm = 0.5f * (ta + tb);
        const float ud = fmaf(fpha, tm - tbase, Fd);
        const float uo = axis_frac(ao, tm);
        const float uz = axis_frac(az, tm);
        const int cd = Idk + __float2int_rd(ud);
        const int co = ao.I + __float2int_rd(uo);
        const int cz = az.I + __float2int_rd(uz);
        const float vd = (float)Idk + ud;
        const float vo = (float)ao.I + uo;
        const int cx = d ? co : cd;
        const int cy = d ? cd : co;
        const int ix = trunc_index(nxm + cx, P.N);
        const int iy = trunc_index(nym - 1 - cy, P.N);
        const int iz = dirz ? trunc_index(nzm - 1 - cz, P.Z) : izflat;
        if ((ix | iy | iz) < 0) return;
        if (!(fmaf(vd, vd, vo * vo) < R2)) return;
        visit((iy * P.N + ix) * P.Z + iz, fabsf(tb - ta));
    };

    const int kcap = Khi;
    for (int k = ks; k <= kcap; k++) {
        const float tk = (float)k;
        const float t0 = tk - 1.0f;
        const int Idk = Id0 + R.pha * (k - 1);
        const bool eo = to_next <= tk;
        const bool ez = tz_next <= tk;
        float tY = 0.0f, tZ = 0.0f;
        if (eo) {
            tY = to_next;
            ao.I = mo; ao.F = 0.0f; ao.ta = tY;
            mo += diro;
            to_next = cross_t(R.O0, invO1, mo);
        }
        if (ez) {
            // the reference splits only at the last z plane crossed in a step
            int guard = 0;
            do {
                tZ = tz_next;
                az.I = mz; az.F = 0.0f; az.ta = tZ;
                mz += dirz;
                if (mz == 0) mz += dirz;
                tz_next = cross_t(R.Z0, invZ1, mz);
            } while (tz_next <= tk && ++guard < 64);
        }
        // order of the split points: the one farther from the step point first
        // (chz > chy, :249-404)
        int ns = 0;
        float a1 = tk, a2 = tk;
        if (eo && ez) {
            const float dY = tk - tY, dZ = tk - tZ;
            if (dZ > dY) { a1 = tZ; a2 = tY; ns = 2; }
            else if (dZ < dY) { a1 = tY; a2 = tZ; ns = 2; }
        } else if (eo) {
            if (tY != tk) { a1 = tY; ns = 1; }
        } else if (ez) {
            if (tZ != tk) { a1 = tZ; ns = 1; }
        }
        segment(t0, ns > 0 ? a1 : tk, t0, Idk);
        if (ns > 0) segment(a1, ns > 1 ? a2 : tk, t0, Idk);
        if (ns > 1) segment(a2, tk, t0, Idk);
    }
}

// -------------------------------------------------------------- visitors --
// Partial sums are kept as pairs of floats and updated with Blackwell's
// packed f32x2 add / fma (one instruction for two elements, each element
// rounded exactly as the scalar fmaf / fadd would round it).
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 f2pack(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2unpack(f32x2 r, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ f32x2 fadd2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 ffma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 fmul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Both uint16 halves of a packed word as exact floats {low, high} without
// the conversion unit: each half is placed in the mantissa of 2^23
// (0x4B000000 | u, a byte permute) and 2^23 is subtracted (exact).
__device__ __forceinline__ f32x2 u16pair(unsigned w)
{
    const float lo = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7410));
    const float hi = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7432));
    return fadd2(f2pack(lo, hi), 0xCB000000CB000000ull);  // {-2^23, -2^23}
}

// Two-level sums: segments accumulate into the pairs P2 (element 2i in the
// low half, 2i+1 in the high half); fold() adds them into L every 32
// iterations, which bounds the FP32 error growth.  The marches pass each
// segment's length in units of the ray parameter (dt); fold() scales the
// pair sums by the ray's cm per unit (lt): one multiply per 32 steps instead
// of one per segment.  first() adds a segment of absolute length to L.
// L lies in shared memory (this thread's column of an [M][threads
// of the block] array): L is touched once per 32 steps, and its registers are
// free for the walk and the interval production.  Sized by the block (not by
// the largest block) so that the shared memory the resident blocks leave to
// L1 is as large as it can be.
__device__ __forceinline__ int ls_stride() { return (int)(blockDim.x * blockDim.y); }
template <int M>
struct PairSums {
    static constexpr int NP = (M + 1) / 2;
    float* Ls;
    f32x2 P2[NP];
    float lt = 1.0f;
    __device__ __forceinline__ float Lget(int i) const { return Ls[i * ls_stride()]; }
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int i = 0; i < M; i++) Ls[i * ls_stride()] = 0.0f;
#pragma unroll
        for (int i = 0; i < NP; i++) P2[i] = 0ull;
    }
    __device__ __forceinline__ void fold()
    {
#pragma unroll
        for (int i = 0; i < NP; i++) {
            float a, b;
            f2unpack(P2[i], a, b);
            Ls[2 * i * ls_stride()] = fmaf(a, lt, Ls[2 * i * ls_stride()]);
            if (2 * i + 1 < M) Ls[(2 * i + 1) * ls_stride()] = fmaf(b, lt, Ls[(2 * i + 1) * ls_stride()]);
            P2[i] = 0ull;
        }
    }
    __device__ __forceinline__ void zero_L()
    {
#pragma unroll
        for (int i = 0; i < M; i++) Ls[i * ls_stride()] = 0.0f;
    }
};

template <int M, bool PIPE = false>
struct AccumU16 : PairSums<M> {
    const uint4* __restrict__ vol;
    __device__ __forceinline__ AccumU16(const uint4* v, float* ls) : vol(v)
    {
        this->Ls = ls;
        this->clear();
        if constexpr (PIPE) {
            pend = none();
            plen = 0.0f;
        }
    }
    // called by all 32 lanes together; p: this lane has a segment
    __device__ __forceinline__ void lanes(bool p, int idx, float len)
    {
        if (p) (*this)(idx, len);
    }
    typedef uint4 Rec;  // one voxel record as loaded
    Rec pend;
    float plen;
    static constexpr int kStride = 1;  // uint4 of a record
    static __device__ __forceinline__ Rec load_at(const uint4* p) { return __ldg(p); }
    __device__ __forceinline__ Rec load(int idx) const { return load_at(vol + idx); }
    static __device__ __forceinline__ Rec none() { return make_uint4(0u, 0u, 0u, 0u); }
    static constexpr bool kFinite = true;  // any record times 0 adds 0
    // P += record * {len, len}
    static __device__ __forceinline__ void add(f32x2 (&P)[PairSums<M>::NP], const Rec& v, f32x2 l2)
    {
        P[0] = ffma2(u16pair(v.x), l2, P[0]);
        P[1] = ffma2(u16pair(v.y), l2, P[1]);
        P[2] = ffma2(u16pair(v.z), l2, P[2]);
        if (M > 6) P[3 % PairSums<M>::NP] = ffma2(u16pair(v.w), l2, P[3 % PairSums<M>::NP]);
    }
    // PIPE: a record is added when the next one has been asked for, so that the
    // lane's gathers overlap (the order of the sums stays)
    __device__ __forceinline__ void operator()(int idx, float len)
    {
        if constexpr (PIPE) {
            drain();
            pend = load(idx);
            plen = len;
        } else {
            add(this->P2, load(idx), f2pack(len, len));
        }
    }
    __device__ __forceinline__ void drain() { add(this->P2, pend, f2pack(plen, plen)); }
    // before the pair sums are folded
    __device__ __forceinline__ void settle()
    {
        if constexpr (PIPE) {
            drain();
            plen = 0.0f;
            pend = none();
        }
    }
    // a segment of absolute length len (cm), straight into L
    __device__ __forceinline__ void first(int idx, float len)
    {
        const uint4 v = __ldg(vol + idx);
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < M; i++) {
            float a, b;
            f2unpack(u16pair(w[i / 2]), a, b);
            this->Ls[i * ls_stride()] = fmaf((i & 1) ? b : a, len, this->Ls[i * ls_stride()]);
        }
    }
};

template <int M, bool PIPE = false>
struct AccumF32 : PairSums<M> {
    using Base = PairSums<M>;
    const uint4* __restrict__ vol;
    __device__ __forceinline__ AccumF32(const uint4* v, float* ls) : vol(v)
    {
        this->Ls = ls;
        this->clear();
        if constexpr (PIPE) {
            pend = none();
            plen = 0.0f;
        }
    }
    __device__ __forceinline__ void lanes(bool p, int idx, float len)
    {
        if (p) (*this)(idx, len);
    }
    struct Rec {  // one voxel record as loaded
        ulonglong2 a, b;
    };
    Rec pend;
    float plen;
    static constexpr int kStride = 2;
    static __device__ __forceinline__ Rec load_at(const uint4* p)
    {
        Rec r;  // the whole record in one 32-byte load
        asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
            : "=l"(r.a.x), "=l"(r.a.y), "=l"(r.b.x), "=l"(r.b.y)
            : "l"(p));
        return r;
    }
    // the walk reads a record as two halves: 4 % faster than one 32-byte load
    // where every lane reads its own (448x448x120, 100 x 100 x 60 views)
    __device__ __forceinline__ Rec load(int idx) const
    {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(vol + 2 * (size_t)idx);
        return Rec{__ldg(p), __ldg(p + 1)};
    }
    static __device__ __forceinline__ Rec none()
    {
        return Rec{make_ulonglong2(0ull, 0ull), make_ulonglong2(0ull, 0ull)};
    }
    static constexpr bool kFinite = false;  // infinities and NaN are values too
    // P += record * {len, len}
    static __device__ __forceinline__ void add(f32x2 (&P)[Base::NP], const Rec& v, f32x2 l2)
    {
        P[0] = ffma2(v.a.x, l2, P[0]);
        P[1] = ffma2(v.a.y, l2, P[1]);
        P[2] = ffma2(v.b.x, l2, P[2]);
        if (M > 6) P[3 % Base::NP] = ffma2(v.b.y, l2, P[3 % Base::NP]);
    }
    // PIPE: a record is added when the next one has been asked for, so that the
    // lane's gathers overlap (the order of the sums stays)
    __device__ __forceinline__ void operator()(int idx, float len)
    {
        if constexpr (PIPE) {
            drain();
            pend = load(idx);
            plen = len;
        } else {
            add(this->P2, load(idx), f2pack(len, len));
        }
    }
    __device__ __forceinline__ void drain() { add(this->P2, pend, f2pack(plen, plen)); }
    // before the pair sums are folded
    __device__ __forceinline__ void settle()
    {
        if constexpr (PIPE) {
            drain();
            plen = 0.0f;
            pend = none();
        }
    }
    // a segment of absolute length len (cm), straight into L
    __device__ __forceinline__ void first(int idx, float len)
    {
        const float* p = reinterpret_cast<const float*>(vol + 2 * (size_t)idx);
#pragma unroll
        for (int i = 0; i < M; i++) {
            this->Ls[i * ls_stride()] = fmaf(__ldg(p + i), len, this->Ls[i * ls_stride()]);
        }
    }
};

// Scatter of one segment's gradient into element planes: plane k holds
// element k of every voxel at the packed record index (y*N + x)*Z + z, so
// the 32 lanes of a warp -- adjacent detector rows, adjacent z cells of one
// xy cell -- reduce into a few consecutive sectors of each plane (one
// reduction per element and lane; the L2 applies them per sector).
template <int M>
struct Scatter {
    float* __restrict__ grad;   // element groups: quads [N*N*Z][4] (elements 4q .. 4q+3), the last
                                // group a pair [N*N*Z][2] when it holds one or two elements
    size_t plane;               // N*N*Z
    int nmat;
    float g[8];                 // zero beyond nmat
    unsigned lo, span;          // packed indices [lo, lo + span) of the strip scattered into
    float lt;                   // cm per unit of the ray parameter (the march passes dt)
    __device__ __forceinline__ void operator()(int idx, float dt) { first(idx, dt * lt); }
    // a segment of absolute length len (cm)
    __device__ __forceinline__ void first(int idx, float len)
    {
        if ((unsigned)idx - lo >= span) return;
        float v[M];
#pragma unroll
        for (int i = 0; i < M; i++) v[i] = g[i] * len;
        add(idx, v);
    }
    // v (zero beyond nmat) added to a voxel: one 16-byte vector reduction per
    // group of four elements (8 bytes for a last group of one or two): a third
    // fewer reduction requests than per element pair for six elements, the
    // same sectors
    __device__ __forceinline__ void add(int idx, const float (&v)[M]) const
    {
#pragma unroll
        for (int q = 0; q < (M + 3) / 4; q++) {
            const int e0 = 4 * q;
            if (e0 >= nmat) break;
            float* base = grad + (size_t)e0 * plane;  // earlier groups are full quads
            if (nmat - e0 > 2)
                atomicAdd(reinterpret_cast<float4*>(base) + idx,
                          make_float4(v[e0], v[e0 + 1], v[(e0 + 2) % M], v[(e0 + 3) % M]));
            else
                atomicAdd(reinterpret_cast<float2*>(base) + idx, make_float2(v[e0], v[e0 + 1]));
        }
    }
    __device__ __forceinline__ void lanes(bool p, int idx, float len)
    {
        if (p) (*this)(idx, len);
    }
};

// ------------------------------------------------- interval march (fast) --
// The xy part of a ray's segments is the same for the 32 rays of a warp (one
// detector column): the dominant-axis steps cut by the crossings of the other
// in-plane axis.  Every 32 steps the lanes compute those xy intervals in
// parallel (lane l takes step k0 + l: its o-plane crossing, each piece's xy
// cell and cylinder test, all in FP64), a warp scan packs them into shared
// memory, and then every lane walks the list with only its own z work: a
// cached slice index, and an exact slow path at the rare z-plane crossings.
// The segments are those of the per-step march whenever at most one z plane
// is crossed per step (|Z1| < 1); warps with steeper rays use the per-step
// march, which reproduces the reference's last-plane-only split.
struct IvRec {
    float ta, tb;  // parameter range of the xy interval
    int base;      // (iy*N + ix)*Z of its midpoint, or -1 (outside mask / bounds)
    float lim;     // ta if every sub-segment has the same xy cell and mask result, else tb:
                   // a z crossing at or before lim needs the exact path
};

constexpr int kIvPerWarp = 64;

// The xy part of the ray plan: identical for the 32 rays of a warp (one
// detector column), so it is kept once per warp in shared memory after the
// interval buffer instead of in every lane's registers.  The interval
// producer and the slow path read it from there.
struct XyPlan {
    double D0, O0, O1, invO1, tc0, tc1;
    int pha, d;
    int dint;  // D0 is an integer: no dominant-axis plane lies inside a step
};
// Interval i lies at slot iv_slot(i): a gap after every four, so that lanes
// reading the same place of different chunks (of four, eight or sixteen)
// meet in different banks.
__device__ __host__ constexpr int iv_slot(int i) { return i + (i >> 2); }
// The walk's own lists have no gaps: all its lanes read one interval at a
// time, and what the buffers leave of the SM's 256 KB is L1.
__device__ __host__ constexpr int plan_slot(bool gaps) { return gaps ? iv_slot(kIvPerWarp) : kIvPerWarp; }
__device__ __host__ constexpr int iv_slots(bool gaps)
{
    return plan_slot(gaps) + (int)((sizeof(XyPlan) + sizeof(IvRec) - 1) / sizeof(IvRec));
}

// An interval as the column sums read it.
struct ColRec {
    unsigned long long len;  // its length twice (a float pair), 0: no voxel
    int base;                // 0 where there is no voxel
    int pad;
};

template <bool GAPS>
__device__ __forceinline__ const XyPlan& publish_plan(const RayPlan& R, IvRec* wbuf)
{
    XyPlan* xp = reinterpret_cast<XyPlan*>(wbuf + plan_slot(GAPS));
    if (threadIdx.x == 0 && R.active) {
        xp->D0 = R.D0;
        xp->O0 = R.O0;
        xp->O1 = R.O1;
        xp->invO1 = R.invO1;
        xp->tc0 = R.tc0;
        xp->tc1 = R.tc1;
        xp->pha = R.pha;
        xp->d = R.d;
        xp->dint = R.D0 == floor(R.D0);
    }
    __syncwarp();
    return *xp;
}

// xy cell of the point at parameter t (FP64), as the reference's midpoint
// rule: -1 when outside the cylindrical mask or the volume.
__device__ __forceinline__ int xy_base_at(const ProjParams& P, const XyPlan& R, double t)
{
    const int nxm = (int)(P.N * 0.5), nym = (int)(P.N * 0.5);
    const double Rv = P.N * 0.5;
    const double Dm = R.D0 + R.pha * t, Om = R.O0 + R.O1 * t;
    if (!(Dm * Dm + Om * Om < Rv * Rv)) return -1;
    const int cd = (int)floor(Dm), co = (int)floor(Om);
    const int cx = R.d ? co : cd, cy = R.d ? cd : co;
    const int ix = trunc_index(nxm + cx, P.N), iy = trunc_index(nym - 1 - cy, P.N);
    if (ix < 0 || iy < 0) return -1;
    return (iy * P.N + ix) * P.Z;
}

__device__ __forceinline__ bool make_rec(const ProjParams& P, const XyPlan& R, double ta,
                                         double tb, IvRec& rec)
{
    // keep every interval that meets the mask chord: a z split can move a
    // sub-segment's midpoint inside even when the interval's is outside
    if (!(tb > R.tc0 - 1e-9 && ta < R.tc1 + 1e-9)) return false;
    rec.ta = (float)ta;
    rec.tb = (float)tb;
    if (!(rec.tb > rec.ta)) return false;  // zero-length (a crossing exactly at a step)
    rec.base = xy_base_at(P, R, 0.5 * (ta + tb));
    // a dominant-axis plane strictly inside (only when 1/s is not an integer)
    // or the mask boundary inside makes sub-segments' cells differ
    bool dplane = false;
    if (!R.dint) {
        const double da = R.D0 + R.pha * ta, db = R.D0 + R.pha * tb;
        const double lo = fmin(da, db), hi = fmax(da, db);
        double m = floor(hi);
        if (m == hi) m -= 1.0;
        dplane = m > lo;
    }
    const bool edge = (R.tc0 > ta && R.tc0 < tb) || (R.tc1 > ta && R.tc1 < tb);
    rec.lim = (dplane || edge) ? rec.tb : rec.ta;
    return true;
}

// Intervals of steps [k0, min(k0 + 31, Khi)] into buf; returns their number.
// off: the place of the first interval of this lane's step (or of the next
// one made, where the step has none).  COL: the column records rec too.
template <bool COL>
__device__ __forceinline__ int produce_intervals(const ProjParams& P, const XyPlan& R, int k0,
                                                 int Khi, IvRec* buf, ColRec* rec, int& off)
{
    const int lane = threadIdx.x;
    const int k = k0 + lane;
    IvRec r0, r1;
    bool v0 = false, v1 = false;
    if (k <= Khi) {
        const double tk = (double)k, tkm = tk - 1.0;
        double tsplit = tk;
        bool ev = false;
        if (R.O1 != 0.0) {
            // a plane m of the other axis is crossed in (k-1, k]: floor changes
            // (all integers, the zero plane included: reprojectionOnGPU.cu:226)
            const double fk = floor(R.O0 + R.O1 * tk), fkm = floor(R.O0 + R.O1 * tkm);
            if (fk != fkm) {
                const double m = (R.O1 > 0.0) ? fk : fkm;
                const double t = (m - R.O0) * R.invO1;
                if (t > tkm && t < tk) {
                    ev = true;
                    tsplit = t;
                }
            }
        }
        v0 = make_rec(P, R, tkm, tsplit, r0);
        if (ev) v1 = make_rec(P, R, tsplit, tk, r1);
    }
    const unsigned b0 = __ballot_sync(0xffffffffu, v0), b1 = __ballot_sync(0xffffffffu, v1);
    const unsigned lt = (1u << lane) - 1u;
    off = __popc(b0 & lt) + __popc(b1 & lt);
    const int total = __popc(b0) + __popc(b1);
    auto put = [&](int i, const IvRec& r) {
        buf[COL ? iv_slot(i) : i] = r;
        if (COL) {
            const float len = r.base >= 0 ? r.tb - r.ta : 0.0f;
            rec[iv_slot(i)] = ColRec{f2pack(len, len), max(r.base, 0), 0};
        }
    };
    if (v0) put(off, r0);
    if (v1) put(off + (int)v0, r1);
    if (COL && lane < 16) {  // the last chunk's places past the list: no voxel
        rec[iv_slot(total + lane)] = ColRec{0ull, 0, 0};
        if (total + lane < kIvPerWarp) buf[iv_slot(total + lane)] = IvRec{0.0f, 0.0f, -1, 0.0f};
    }
    __syncwarp();
    return total;
}

// Per-lane z state of the interval march.
struct ZState {
    int cz;        // floor(z / step) of the current position's cell
    int iz;        // its slice index (trunc rule), or -1
    int mz;        // next z plane that splits (never 0: :237-238)
    int dirz;
    float tz_next; // parameter of that crossing
    float tz0;     // parameter of the (non-splitting) z = 0 crossing ahead, or inf
};

__device__ __forceinline__ float zcross(const RayPlan& R, int m)
{
    return (float)(((double)m - R.Z0) * R.invZ1);
}

__device__ __forceinline__ void zstate_init(const ProjParams& P, const RayPlan& R, double t0, ZState& z)
{
    const int nzm = (int)(P.Z * 0.5);
    const double v = R.Z0 + R.Z1 * t0;
    const double fl = floor(v);
    z.cz = (int)fl;
    z.dirz = (R.Z1 > 0.0) ? 1 : ((R.Z1 < 0.0) ? -1 : 0);
    z.tz_next = kInf;
    z.tz0 = kInf;
    if (z.dirz) {
        z.mz = (z.dirz > 0) ? z.cz + 1 : ((v == fl) ? z.cz - 1 : z.cz);
        if (z.mz == 0) z.mz += z.dirz;
        z.tz_next = zcross(R, z.mz);
        if ((z.dirz > 0 && v < 0.0) || (z.dirz < 0 && v > 0.0)) z.tz0 = zcross(R, 0);
        z.iz = trunc_index(nzm - 1 - z.cz, P.Z);
    } else {
        z.iz = flat_z_index(P, R.Z0);
    }
}

// One interval, exact: split it at the z planes inside it (and apply the
// midpoint rule across the z = 0 plane, which does not split).
template <class Visit>
__device__ __forceinline__ void consume_slow(const ProjParams& P, const RayPlan& R, const XyPlan& xp,
                                             const IvRec& rc,
                                             ZState& z, Visit& visit)
{
    const int nzm = (int)(P.Z * 0.5);
    float cur = rc.ta;
    const float tb = rc.tb;
    // crossings in intervals that were not produced (outside the mask chord)
    // only move the state
    for (int guard = 0; z.tz_next <= cur && guard < 64; guard++) {
        z.cz = (z.dirz > 0) ? z.mz : z.mz - 1;
        z.mz += z.dirz;
        if (z.mz == 0) z.mz += z.dirz;
        z.tz_next = zcross(R, z.mz);
    }
    if (z.tz0 <= cur) {
        z.cz = (z.dirz > 0) ? 0 : -1;
        z.tz0 = kInf;
    }
    for (int guard = 0; guard < 8; guard++) {
        const bool split = z.tz_next <= tb;
        const float end = split ? z.tz_next : tb;
        int cseg = z.cz;
        if (z.tz0 <= end) {
            const int after = (z.dirz > 0) ? 0 : -1;
            if (0.5f * (cur + end) >= z.tz0) cseg = after;
            z.cz = after;
            z.tz0 = kInf;
        }
        if (end > cur) {
            const bool whole = (cur == rc.ta) && (end == tb);
            const int base = whole ? rc.base : xy_base_at(P, xp, 0.5 * ((double)cur + (double)end));
            const int iz = trunc_index(nzm - 1 - cseg, P.Z);
            if (base >= 0 && iz >= 0) visit(base + iz, end - cur);
        }
        if (!split) break;
        z.cz = (z.dirz > 0) ? z.mz : z.mz - 1;
        cur = end;
        z.mz += z.dirz;
        if (z.mz == 0) z.mz += z.dirz;
        z.tz_next = zcross(R, z.mz);
    }
    z.iz = trunc_index(nzm - 1 - z.cz, P.Z);
}

template <class Visit>
__device__ __forceinline__ void consume_one(const ProjParams& P, const RayPlan& R, const XyPlan& xp,
                                            const IvRec& rc,
                                            ZState& z, Visit& visit)
{
    if (z.tz_next <= rc.tb || z.tz0 <= rc.tb) {
        consume_slow(P, R, xp, rc, z, visit);
    } else if (rc.base >= 0 && z.iz >= 0) {
        visit(rc.base + z.iz, rc.tb - rc.ta);
    }
}

// A batch of intervals, each ray on its own, the warp interval by interval.
// Per interval the common case is one vector load in the lane's current z
// cell; a z crossing inside an exact interval splits it inline (second load
// in the new cell).  Everything else -- the non-splitting z = 0 plane, a
// crossing in an interval whose sub-segments may change xy cell or mask
// result, and crossings passed in intervals that were not produced -- goes
// through consume_slow.  Both branches are taken warp-uniformly.
template <bool COL, class Visit>
__device__ __forceinline__ void walk_batch(const ProjParams& P, const RayPlan& R, const XyPlan& xp, const IvRec* buf,
                                           int total, ZState& z, Visit& visit)
{
    const int nzm = (int)(P.Z * 0.5);
    // one interval per loop trip: two spill more than they overlap (200x200x60
    // views of 64x64x16: 0.456 ms against 0.481)
#pragma unroll 1
    for (int i = 0; i < total; i++) {
        const IvRec rc = buf[COL ? iv_slot(i) : i];
        const bool rare = (z.tz0 <= rc.tb) || (z.tz_next <= rc.lim);
        if (__any_sync(0xffffffffu, rare)) {
            consume_one(P, R, xp, rc, z, visit);
            continue;
        }
        const bool ev = z.tz_next <= rc.tb;
        const float tz = ev ? z.tz_next : rc.tb;
        visit.lanes(rc.base >= 0 && z.iz >= 0, rc.base + z.iz, tz - rc.ta);
        if (__any_sync(0xffffffffu, ev)) {
            if (ev) {
                z.cz = (z.dirz > 0) ? z.mz : z.mz - 1;
                z.iz = trunc_index(nzm - 1 - z.cz, P.Z);
                z.mz += z.dirz;
                if (z.mz == 0) z.mz += z.dirz;
                z.tz_next = zcross(R, z.mz);
            }
            visit.lanes(ev && rc.base >= 0 && z.iz >= 0 && rc.tb > tz, rc.base + z.iz, rc.tb - tz);
        }
    }
}

// Inactive lanes follow the warp without contributing.
__device__ __forceinline__ void zstate_start(const ProjParams& P, const RayPlan& R, bool act, int Klo, ZState& z)
{
    zstate_init(P, R, (double)(Klo - 1), z);
    if (!act) {
        z.iz = -1;
        z.tz_next = kInf;
        z.tz0 = kInf;
    }
}

// Iterations [Klo, Khi] of one ray by intervals; `flush` folds partial sums.
template <class Visit, class Flush>
__device__ __forceinline__ void march_intervals(const ProjParams& P, const RayPlan& R, const XyPlan& xp, bool act,
                                                int Klo, int Khi, IvRec* buf, Visit& visit,
                                                Flush flush)
{
    ZState z;
    zstate_start(P, R, act, Klo, z);
    for (int k0 = Klo; k0 <= Khi; k0 += 32) {
        int off;
        const int total = produce_intervals<false>(P, xp, k0, Khi, buf, nullptr, off);
        walk_batch<false>(P, R, xp, buf, total, z, visit);
        __syncwarp();
        flush();
    }
}

// ------------------------------------------------- column march (shared) --
// The rays of a warp that lie in one slice read the same voxel records: with
// slices thicker than the detector pitch at the volume, ~3 of the 32 lanes
// share each record, and along a batch of steps most rays stay in one slice.
// So the sums along the batch are made once per slice and not once per ray:
// the batch's intervals are cut into chunks, every lane takes a (chunk,
// slice) pair at a time and sums length x record down the chunk --
// independent loads, no slice bookkeeping -- into shared memory; then every
// ray adds, chunk by chunk, the sums of the slice it is in, and walks on its
// own only the chunk in which it meets a z plane.
constexpr int kColEntries = 160;  // (chunk, slice) pairs of a batch
template <int M>
struct ColTab {
    ColRec rec[iv_slot(kIvPerWarp + 16)];
    float4 a[kColEntries];                                       // elements 0-3
    std::conditional_t<(M > 6), float4, float2> b[kColEntries];  // 4, 5 (6, 7)
};

// Pair p = chunk * cells + cell: intervals [chunk << lg, (chunk + 1) << lg),
// slice zb + cell.
template <class Acc, int M>
__device__ __forceinline__ void column_sums(const Acc& acc, int nch, int lg, int zb, int cells, ColTab<M>* tab)
{
    constexpr int NP = (M + 1) / 2;
    const int pairs = nch * cells;
    // pair p + 32 lies dc chunks and dz slices on
    const float rcells = __frcp_rn((float)cells);
    const int dc = __float2int_rd(32.5f * rcells), dz = 32 - dc * cells;
    int c = __float2int_rd(((float)threadIdx.x + 0.5f) * rcells);
    int cell = threadIdx.x - c * cells;
    const uint4* vol0 = acc.vol + (size_t)zb * Acc::kStride;
    for (int p = threadIdx.x; p < pairs; p += 32) {
        const uint4* col = vol0 + cell * Acc::kStride;
        const ColRec* b = tab->rec + iv_slot(c << lg);
        f32x2 S[NP];
#pragma unroll
        for (int i = 0; i < NP; i++) S[i] = 0ull;
#pragma unroll 1
        for (int i0 = 0; i0 < (1 << lg); i0 += 4, b += iv_slot(4)) {
            ColRec r[4];
            typename Acc::Rec v[4];
#pragma unroll
            for (int i = 0; i < 4; i++) r[i] = b[i];
            if (Acc::kFinite || (r[0].len && r[1].len && r[2].len && r[3].len)) {
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = Acc::load_at(col + (size_t)(unsigned)r[i].base * Acc::kStride);
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    v[i] = Acc::none();
                    if (r[i].len) v[i] = Acc::load_at(col + (size_t)(unsigned)r[i].base * Acc::kStride);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) Acc::add(S, v[i], r[i].len);
        }
        *reinterpret_cast<ulonglong2*>(tab->a + p) = make_ulonglong2(S[0], S[1]);
        if constexpr (M > 6) *reinterpret_cast<ulonglong2*>(tab->b + p) = make_ulonglong2(S[2], S[3 % NP]);
        else *reinterpret_cast<f32x2*>(tab->b + p) = S[2];
        cell += dz;
        c += dc;
        if (cell >= cells) {
            cell -= cells;
            c++;
        }
    }
}

template <class Acc, int M>
__device__ __forceinline__ void column_add(const ColTab<M>* tab, int o, Acc& acc)
{
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(tab->a + o);
    acc.P2[0] = fadd2(acc.P2[0], a.x);
    acc.P2[1] = fadd2(acc.P2[1], a.y);
    if constexpr (M > 6) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(tab->b + o);
        acc.P2[2] = fadd2(acc.P2[2], b.x);
        acc.P2[3 % Acc::NP] = fadd2(acc.P2[3 % Acc::NP], b.y);
    } else {
        acc.P2[2] = fadd2(acc.P2[2], *reinterpret_cast<const f32x2*>(tab->b + o));
    }
}

// One interval of one ray on its own: walk_batch's step without its warp votes.
template <class Visit>
__device__ __forceinline__ void ray_interval(const ProjParams& P, const RayPlan& R, const XyPlan& xp, const IvRec& rc,
                                             ZState& z, Visit& visit)
{
    if (z.tz0 <= rc.tb || z.tz_next <= rc.lim) {
        consume_slow(P, R, xp, rc, z, visit);
        return;
    }
    const bool ev = z.tz_next <= rc.tb;
    const float tz = ev ? z.tz_next : rc.tb;
    if (rc.base >= 0 && z.iz >= 0) visit(rc.base + z.iz, tz - rc.ta);
    if (ev) {
        const int nzm = (int)(P.Z * 0.5);
        z.cz = (z.dirz > 0) ? z.mz : z.mz - 1;
        z.iz = trunc_index(nzm - 1 - z.cz, P.Z);
        z.mz += z.dirz;
        if (z.mz == 0) z.mz += z.dirz;
        z.tz_next = zcross(R, z.mz);
        if (rc.base >= 0 && z.iz >= 0 && rc.tb > tz) visit(rc.base + z.iz, rc.tb - tz);
    }
}

// A ray that meets more than one z plane in the part of the batch (or z = 0,
// or lies outside the table): its chunks in order, the shared sums where it
// meets none, its own walk elsewhere.
template <class Acc, int M>
__device__ __forceinline__ void column_ray(const ProjParams& P, const RayPlan& R, const XyPlan& xp, const IvRec* buf,
                                        int n, int lg, int zb, int cells, const ColTab<M>* tab, ZState& z, Acc& acc)
{
    const int nch = (n + (1 << lg) - 1) >> lg;
    // chunks up to the next one with a plane, then that one: the warp goes
    // round once per plane of its busiest ray
    for (int c = 0; c < nch;) {
        const int cell = z.iz - zb;
        const bool in = z.iz >= 0 && (unsigned)cell < (unsigned)cells;
        const float te = fminf(z.tz_next, z.tz0);
        while (c < nch && (in || z.iz < 0) && te > buf[iv_slot(min((c + 1) << lg, n) - 1)].tb) {
            if (in) column_add<Acc, M>(tab, c * cells + cell, acc);
            c++;
        }
        if (c >= nch) break;
        const int i1 = min((c + 1) << lg, n);
#pragma unroll 1
        for (int i = c << lg; i < i1; i++) {
            const IvRec rc = buf[iv_slot(i)];
            ray_interval(P, R, xp, rc, z, acc);
        }
        c++;
    }
}

// A z plane crossing of a ray in a batch.
struct ZEvent {
    float t;  // its parameter
    int i;    // the interval it is in (the next one, where none was made there)
    int iz;   // slice after it
};

// Up to two z planes that a ray meets in a batch, and the slices it is in.
struct BatchEvents {
    ZState z;       // after them
    int ne;
    ZEvent e1, e2;
    int lo, hi;     // slices (lo > hi: none)
    bool simple;    // it meets no others, nor z = 0
};
__device__ __forceinline__ BatchEvents batch_events(const ProjParams& P, const RayPlan& R, const ZState& z,
                                                    const IvRec* buf, int off, int k0, int total, float tlast)
{
    const int nzm = (int)(P.Z * 0.5);
    BatchEvents b;
    b.z = z;
    b.ne = 0;
    b.e1 = b.e2 = ZEvent{kInf, kIvPerWarp, z.iz};
    b.lo = z.iz >= 0 ? z.iz : INT_MAX;
    b.hi = z.iz;
    // the next crossing: the interval of its step, or the next one made
    auto interval = [&]() -> int {
        const float t = b.z.tz_next;
        const int s = min(max(__float2int_ru(fminf(t, (float)(k0 + 32))) - k0, 0), 31);
        int i = __shfl_sync(0xffffffffu, off, s);
        if (i < total && t > buf[iv_slot(i)].tb) i++;
        return i;
    };
    auto cross = [&](ZEvent& e, int i) {
        ZState& q = b.z;
        e.t = q.tz_next;
        e.i = i;
        q.cz = (q.dirz > 0) ? q.mz : q.mz - 1;
        q.iz = trunc_index(nzm - 1 - q.cz, P.Z);
        q.mz += q.dirz;
        if (q.mz == 0) q.mz += q.dirz;
        q.tz_next = zcross(R, q.mz);
        e.iz = q.iz;
        b.lo = min(b.lo, q.iz >= 0 ? q.iz : INT_MAX);
        b.hi = max(b.hi, q.iz);
        b.ne++;
    };
    {
        const int i = interval();
        if (b.z.tz_next <= tlast) {
            cross(b.e1, i);
            b.e2.iz = b.e1.iz;
        }
    }
    const bool second = b.ne == 1 && b.z.tz_next <= tlast;
    if (__any_sync(0xffffffffu, second)) {
        const int i = interval();
        if (second) cross(b.e2, i);
    }
    b.simple = z.tz0 > tlast && b.z.tz_next > tlast;
    return b;
}

// The chunk of a crossing: whole intervals before and after it, then the two
// pieces of the one it cuts.
template <class Acc>
__device__ __forceinline__ void column_event(const ProjParams& P, const XyPlan& xp, const IvRec* q, int len4,
                                             const ZEvent& e, int iz0, Acc& acc)
{
    int cut = -1;
#pragma unroll 1
    for (int i0 = 0; i0 < len4; i0 += 4) {
        typename Acc::Rec v[4];
        float len[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const IvRec rc = q[iv_slot(i0) + i];
            const bool before = rc.tb <= e.t;
            const int iz = before ? iz0 : e.iz;
            const bool whole = before || rc.ta >= e.t;
            if (!whole) cut = iv_slot(i0) + i;
            const bool use = whole && rc.base >= 0 && iz >= 0;
            len[i] = use ? rc.tb - rc.ta : 0.0f;
            v[i] = Acc::none();
            if (use) v[i] = Acc::load_at(acc.vol + (size_t)(unsigned)(rc.base + iz) * Acc::kStride);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) Acc::add(acc.P2, v[i], f2pack(len[i], len[i]));
    }
    if (cut >= 0) {
        const IvRec rc = q[cut];
        int b1 = rc.base, b2 = rc.base;
        if (e.t <= rc.lim) {  // the pieces may differ in xy cell or mask
            b1 = xy_base_at(P, xp, 0.5 * ((double)rc.ta + (double)e.t));
            b2 = xy_base_at(P, xp, 0.5 * ((double)e.t + (double)rc.tb));
        }
        if (b1 >= 0 && iz0 >= 0) acc(b1 + iz0, e.t - rc.ta);
        if (b2 >= 0 && e.iz >= 0) acc(b2 + e.iz, rc.tb - e.t);
    }
}

template <class Acc, int M, class Flush>
__device__ __forceinline__ void march_columns(const ProjParams& P, const RayPlan& R, const XyPlan& xp, bool act,
                                              int Klo, int Khi, IvRec* buf, ColTab<M>* tab, Acc& acc, Flush flush)
{
    ZState z;
    zstate_start(P, R, act, Klo, z);
    for (int k0 = Klo; k0 <= Khi; k0 += 32) {
        int off;
        const int total = produce_intervals<true>(P, xp, k0, Khi, buf, tab->rec, off);
        if (total == 0) continue;
        const float tlast = buf[iv_slot(total - 1)].tb;
        const BatchEvents ev = batch_events(P, R, z, buf, off, k0, total, tlast);
        const int zb = __reduce_min_sync(0xffffffffu, ev.lo), zh = __reduce_max_sync(0xffffffffu, ev.hi);
        const int cells = zh < 0 ? 0 : zh - zb + 1;
        if (cells > 32) {  // detector pitch above the slices': little is shared
            walk_batch<true>(P, R, xp, buf, total, z, acc);
            __syncwarp();
            flush();
            continue;
        }
        int lg = 2;
        while (cells * ((total + (1 << lg) - 1) >> lg) > kColEntries) lg++;
        const int nch = (total + (1 << lg) - 1) >> lg;
        __syncwarp();
        if (cells > 0) column_sums<Acc, M>(acc, nch, lg, zb, cells, tab);
        __syncwarp();
        const int c1 = ev.e1.i >> lg, c2 = ev.e2.i >> lg;
        if (ev.simple && (ev.ne < 2 || c1 != c2)) {
            int iz = z.iz;
#pragma unroll 2
            for (int c = 0, o = -zb; c < nch; c++, o += cells) {
                if (c == c1 || c == c2) iz = c == c1 ? ev.e1.iz : ev.e2.iz;
                else if (iz >= 0) column_add<Acc, M>(tab, o + iz, acc);
            }
            if (ev.ne > 0) {
                column_event(P, xp, buf + iv_slot(c1 << lg), 1 << lg, ev.e1, z.iz, acc);
                if (ev.ne > 1) column_event(P, xp, buf + iv_slot(c2 << lg), 1 << lg, ev.e2, ev.e1.iz, acc);
            }
            z = ev.z;
        } else {
            column_ray<Acc, M>(P, R, xp, buf, total, lg, zb, cells, tab, z, acc);
        }
        __syncwarp();
        flush();
    }
}

// The same sharing for the adjoint's scatter: along a chunk that a ray spends
// in one slice its gradient goes to the same voxels as its slice mates', so
// their gradients are added first and reduced once.  Every ray marks, per chunk,
// the slice it is in; a lane per (chunk, slice) then adds up the gradients of
// the rays that marked it and scatters the sum down the chunk.
template <int M>
struct ScatterTab {
    ColRec rec[iv_slot(kIvPerWarp + 16)];
    unsigned rays[kColEntries];                             // per (chunk, slice): its rays
    float4 ga[32];                                          // per ray: gradient per unit of t, elements 0-3
    std::conditional_t<(M > 6), float4, float2> gb[32];     // 4, 5 (6, 7)
};

template <int M>
__device__ __forceinline__ void scatter_sums(const Scatter<M>& sc, int nch, int lg, int zb, int cells,
                                             const ScatterTab<M>* tab)
{
    constexpr int NP = (M + 1) / 2;
    const int pairs = nch * cells;
    const float rcells = __frcp_rn((float)cells);
    const int dc = __float2int_rd(32.5f * rcells), dz = 32 - dc * cells;
    int c = __float2int_rd(((float)threadIdx.x + 0.5f) * rcells);
    int cell = threadIdx.x - c * cells;
    for (int p = threadIdx.x; p < pairs; p += 32) {
        unsigned m = tab->rays[p];
        if (m) {
            f32x2 G[NP];
#pragma unroll
            for (int i = 0; i < NP; i++) G[i] = 0ull;
            do {
                const int ray = __ffs(m) - 1;
                m &= m - 1;
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(tab->ga + ray);
                G[0] = fadd2(G[0], a.x);
                G[1] = fadd2(G[1], a.y);
                if constexpr (M > 6) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(tab->gb + ray);
                    G[2] = fadd2(G[2], b.x);
                    G[3 % NP] = fadd2(G[3 % NP], b.y);
                } else {
                    G[2] = fadd2(G[2], *reinterpret_cast<const f32x2*>(tab->gb + ray));
                }
            } while (m);
            const ColRec* b = tab->rec + iv_slot(c << lg);
            for (int i0 = 0; i0 < (1 << lg); i0 += 4, b += iv_slot(4)) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const ColRec r = b[i];
                    if (r.len && (unsigned)r.base - sc.lo < sc.span) {
                        float v[2 * NP];
#pragma unroll
                        for (int q = 0; q < NP; q++) f2unpack(fmul2(G[q], r.len), v[2 * q], v[2 * q + 1]);
                        sc.add(r.base + zb + cell, v);
                    }
                }
            }
        }
        cell += dz;
        c += dc;
        if (cell >= cells) {
            cell -= cells;
            c++;
        }
    }
}

template <int M>
__device__ __forceinline__ void scatter_columns(const ProjParams& P, const RayPlan& R, const XyPlan& xp, bool act,
                                                int Klo, int Khi, IvRec* buf, ScatterTab<M>* tab, Scatter<M>& sc)
{
    const int lane = threadIdx.x;
    tab->ga[lane] = make_float4(sc.g[0] * sc.lt, sc.g[1] * sc.lt, sc.g[2] * sc.lt, sc.g[3] * sc.lt);
    if constexpr (M > 6) tab->gb[lane] = make_float4(sc.g[4] * sc.lt, sc.g[5] * sc.lt, sc.g[6] * sc.lt, sc.g[7] * sc.lt);
    else tab->gb[lane] = make_float2(sc.g[4] * sc.lt, sc.g[5] * sc.lt);
    ZState z;
    zstate_start(P, R, act, Klo, z);
    for (int k0 = Klo; k0 <= Khi; k0 += 32) {
        int off;
        const int total = produce_intervals<true>(P, xp, k0, Khi, buf, tab->rec, off);
        if (total == 0) continue;
        const float tlast = buf[iv_slot(total - 1)].tb;
        const BatchEvents ev = batch_events(P, R, z, buf, off, k0, total, tlast);
        const int zb = __reduce_min_sync(0xffffffffu, ev.lo), zh = __reduce_max_sync(0xffffffffu, ev.hi);
        const int cells = zh < 0 ? 0 : zh - zb + 1;
        if (cells > 32) {
            walk_batch<true>(P, R, xp, buf, total, z, sc);
            __syncwarp();
            continue;
        }
        int lg = 2;
        while (cells * ((total + (1 << lg) - 1) >> lg) > kColEntries) lg++;
        const int nch = (total + (1 << lg) - 1) >> lg;
        for (int p = lane; p < nch * cells; p += 32) tab->rays[p] = 0u;
        __syncwarp();
        const int c1 = ev.e1.i >> lg, c2 = ev.e2.i >> lg;
        if (ev.simple && (ev.ne < 2 || c1 != c2)) {
            int iz = z.iz;
            for (int c = 0, o = -zb; c < nch; c++, o += cells) {
                if (c == c1 || c == c2) iz = c == c1 ? ev.e1.iz : ev.e2.iz;
                else if (iz >= 0) atomicOr(&tab->rays[o + iz], 1u << lane);
            }
            // the chunks of its crossings on its own
            for (int n = 0; n < ev.ne; n++) {
                const int c = n ? c2 : c1, i1 = min((c + 1) << lg, total);
#pragma unroll 1
                for (int i = c << lg; i < i1; i++) ray_interval(P, R, xp, buf[iv_slot(i)], z, sc);
            }
            z = ev.z;
        } else {
            for (int c = 0; c < nch;) {
                const int cell = z.iz - zb;
                const bool in = z.iz >= 0 && (unsigned)cell < (unsigned)cells;
                const float te = fminf(z.tz_next, z.tz0);
                while (c < nch && (in || z.iz < 0) && te > buf[iv_slot(min((c + 1) << lg, total) - 1)].tb) {
                    if (in) atomicOr(&tab->rays[c * cells + cell], 1u << lane);
                    c++;
                }
                if (c >= nch) break;
                const int i1 = min((c + 1) << lg, total);
#pragma unroll 1
                for (int i = c << lg; i < i1; i++) ray_interval(P, R, xp, buf[iv_slot(i)], z, sc);
                c++;
            }
        }
        __syncwarp();
        if (cells > 0) scatter_sums<M>(sc, nch, lg, zb, cells, tab);
        __syncwarp();
    }
}

// How a kernel sums along its rays: each ray on its own, or by shared columns.
enum { kWalk = 0, kColumns = 1 };

// Two-level summation: the visitor accumulates into its pair sums; every 32 iterations
// the partials are folded into L (bounds the FP32 error growth).
template <class Acc, int M>
__device__ __forceinline__ void march_accumulate(const ProjParams& P, const RayPlan& R, int Klo,
                                                 int Khi, Acc& acc)
{
    acc.clear();
    acc.lt = R.Lt;
    if (R.first_idx >= 0) acc.first(R.first_idx, R.first_len);
    for (int k0 = Klo; k0 <= Khi; k0 += 32) {
        const int k1 = min(Khi, k0 + 31);
        march(P, R, k0, k1, acc);
        acc.settle();
        acc.fold();
    }
}

// The spectral table in shared memory: bins in pairs, so that the sums over
// bins run two at a time in packed arithmetic.  A last odd bin is paired with
// itself, half the weight each: whatever its exponential is (0 behind an
// infinite path integral, infinite before one of -inf), the pair's sum is the bin's.
template <int M>
struct SpecPair {
    f32x2 mu[M];
    f32x2 pdf;
    f32x2 floor;  // the spectrum's (it fills the pair to a multiple of 16 bytes: M is even)
};
template <int M>
__host__ __device__ constexpr size_t spec_bytes(int NE) { return (size_t)((NE + 1) / 2) * sizeof(SpecPair<M>); }

template <int M>
__device__ __forceinline__ void load_spectrum(const SpectrumDev& sp, SpecPair<M>* s_sp)
{
    constexpr int W = 2 * (M + 2);  // floats of a pair
    const float* mu = reinterpret_cast<const float*>(sp.mu8);
    float* dst = reinterpret_cast<float*>(s_sp);
    const int n = (sp.NE + 1) / 2 * W;
    for (int i = threadIdx.x + threadIdx.y * blockDim.x; i < n; i += blockDim.x * blockDim.y) {
        const int e0 = 2 * (i / W), e = min(e0 + (i & 1), sp.NE - 1), k = (i % W) >> 1;
        dst[i] = k < M ? mu[8 * e + k] : (k == M ? sp.pdf[1 + e] * (e0 + 1 < sp.NE ? 1.0f : 0.5f) : sp.pdf[0]);
    }
}

template <int M>
__device__ __forceinline__ f32x2 attenuation2(const SpecPair<M>& q, const f32x2 (&L2)[M])
{
    f32x2 T = fmul2(q.mu[0], L2[0]);
#pragma unroll
    for (int k = 1; k < M; k++) T = ffma2(q.mu[k], L2[k], T);
    return T;
}

// 2^x of both halves (the hardware's exponential, results below 2^-126 as 0)
__device__ __forceinline__ f32x2 exp2_2(f32x2 x)
{
    float a, b;
    f2unpack(x, a, b);
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(a));
    asm("ex2.approx.ftz.f32 %0, %0;" : "+f"(b));
    return f2pack(a, b);
}

// sum_E pdf_E exp(-sum_k mu_k(E) L_k).  The exponents are formed for base 2 from
// path integrals scaled by -log2 e (rounded once per ray and element, as L
// itself is), so that a bin's exponential is one instruction.  A bin below 2^-126
// counts as 0, at most 2^-126 of the spectrum's weight in all: from a sum of
// 2^-100 of it (the floor) on that is below a quarter of its last place.  A sum
// under the floor, or one that is not finite (a path integral that only its
// scaling takes beyond the largest float), is done again with expf and L as it is.
// Asking every bin instead did most sums of a body twice: 10 keV bins behind
// 20 cm of water are below 2^-126 (48 phantoms of 64x64xZ: 0.321 -> 0.284 ms;
// 256x256x100, 60 views of 200 x 200: 1.54 -> 1.44).
template <int M>
__device__ __forceinline__ float spectral_sum(const SpecPair<M>* s_sp, int NE, const float* L)
{
    f32x2 L2[M], acc = 0ull;
#pragma unroll
    for (int k = 0; k < M; k++) {
        const float l = L[k] * -1.4426950408889634f;
        L2[k] = f2pack(l, l);
    }
#pragma unroll 2
    for (int e = 0; e < (NE + 1) / 2; e++) {
        const SpecPair<M> q = s_sp[e];
        acc = ffma2(q.pdf, exp2_2(attenuation2<M>(q, L2)), acc);
    }
    float a, b, floor, unused;
    f2unpack(acc, a, b);
    f2unpack(s_sp->floor, floor, unused);
    if (!(a + b >= floor && a + b < kInf)) {
        acc = 0ull;
#pragma unroll
        for (int k = 0; k < M; k++) L2[k] = f2pack(L[k], L[k]);
#pragma unroll 1
        for (int e = 0; e < (NE + 1) / 2; e++) {
            const SpecPair<M> q = s_sp[e];
            f2unpack(attenuation2<M>(q, L2), a, b);
            acc = ffma2(q.pdf, f2pack(expf(-a), expf(-b)), acc);
        }
        f2unpack(acc, a, b);
    }
    return a + b;
}

// Warp-uniform iteration range: the union over the warp's lanes.
__device__ __forceinline__ void warp_range(const RayPlan& R, bool valid, int& Klo, int& Khi)
{
    const int lo = (valid && R.active) ? R.klo : INT_MAX;
    const int hi = (valid && R.active) ? R.khi : -1;
    Klo = __reduce_min_sync(0xffffffffu, lo);
    Khi = __reduce_max_sync(0xffffffffu, hi);
}

// Iterations [klo, khi] narrowed to those whose segments can lie in volume
// rows iy in [y0, y1): the ray's y cell cy = floor(D or O) is linear in t
// (iy = nym - 1 - cy), two cells of margin each way; the interval march
// computes every step's cells from t alone, so a narrowed range gives the
// same segments as the whole ray.
__device__ __forceinline__ void strip_iterations(const ProjParams& P, const RayPlan& R, int y0, int y1, int& klo,
                                                 int& khi)
{
    const int nym = (int)(P.N * 0.5);
    const double ca = (double)(nym - y1 - 2), cb = (double)(nym - y0 + 2);  // cy range, with margin
    double ta, tb;
    if (R.d) {                       // y dominant: cy = floor(D0 + pha t)
        ta = (ca - R.D0) * R.pha;
        tb = (cb - R.D0) * R.pha;
    } else if (R.O1 != 0.0) {        // cy = floor(O0 + O1 t)
        ta = (ca - R.O0) * R.invO1;
        tb = (cb - R.O0) * R.invO1;
    } else {                         // constant y
        if (!(R.O0 >= ca && R.O0 <= cb)) khi = klo - 1;
        return;
    }
    if (ta > tb) {
        const double t = ta;
        ta = tb;
        tb = t;
    }
    if (!(tb >= (double)(klo - 1)) || !(ta <= (double)khi)) {
        khi = klo - 1;
        return;
    }
    klo = max(klo, (int)floor(ta));
    khi = min(khi, (int)ceil(tb) + 1);
}

__device__ __forceinline__ void warp_range_k(int klo, int khi, bool use, int& Klo, int& Khi)
{
    Klo = __reduce_min_sync(0xffffffffu, use && klo <= khi ? klo : INT_MAX);
    Khi = __reduce_max_sync(0xffffffffu, use && klo <= khi ? khi : -1);
}

// grid: (ceil(W / cols_per_block), ceil(H / 32), V); block: (32, cols_per_block).
// Per-element path integrals of one ray (first segment + iterations
// [Klo, Khi]).  The interval march is used unless a lane of the warp has
// |Z1| >= 1 (more than one z plane per step), where the per-step march keeps
// the reference's last-plane-only split.  R.active is warp-uniform.
// tab: the warp's column table (kColumns).
template <class Acc, int M, int MODE>
__device__ __forceinline__ void ray_integrals(const ProjParams& P, const RayPlan& R, bool act, int Klo, int Khi,
                                              IvRec* wbuf, Acc& acc, ColTab<M>* tab)
{
    acc.clear();
    if (!R.active) return;
    const bool steep = __any_sync(0xffffffffu, fabs(R.Z1) >= 1.0);
    if (steep) {
        march_accumulate<Acc, M>(P, R, Klo, Khi, acc);
        if (!act) acc.zero_L();
        return;
    }
    acc.lt = R.Lt;
    if (act && R.first_idx >= 0) acc.first(R.first_idx, R.first_len);
    auto fold = [&]() {
        acc.settle();
        acc.fold();
    };
    const XyPlan& xp = publish_plan<MODE != kWalk>(R, wbuf);
    if (Klo <= Khi) {
        if constexpr (MODE == kColumns)
            march_columns<Acc, M>(P, R, xp, act, Klo, Khi, wbuf, tab, acc, fold);
        else
            march_intervals(P, R, xp, act, Klo, Khi, wbuf, acc, fold);
    }
    fold();
}


__device__ __forceinline__ bool is_u16(const VolRef& v) { return (v.form ? *v.form : v.expect) == kFormU16; }

// Counts the segments of a ray that walks; reads no volume.
struct SegmentCount {
    unsigned nseg = 0u;
    float lt;
    __device__ __forceinline__ void operator()(int, float) { nseg++; }
    __device__ __forceinline__ void first(int, float) { nseg++; }
    __device__ __forceinline__ void lanes(bool p, int, float) { nseg += p; }
    __device__ __forceinline__ void clear() {}
    __device__ __forceinline__ void settle() {}
    __device__ __forceinline__ void fold() {}
    __device__ __forceinline__ void zero_L() {}
};

// Path integrals of one ray.
template <int M, int MODE, bool U16>
__device__ __forceinline__ void ray_path(const VolRef& vol, const ProjParams& P, const RayPlan& R, bool act, int Klo,
                                         int Khi, IvRec* wbuf, float* s_L, ColTab<M>* tab, float (&L)[M])
{
    typedef std::conditional_t<U16, AccumU16<M, MODE == kWalk>, AccumF32<M, MODE == kWalk>> Acc;
    Acc acc(static_cast<const uint4*>(vol.rec), s_L);
    ray_integrals<Acc, M, MODE>(P, R, act, Klo, Khi, wbuf, acc, tab);
#pragma unroll
    for (int i = 0; i < M; i++) L[i] = acc.Lget(i);
}

// One work tile of the forward projection: detector columns
// [colb*cpb, colb*cpb + cpb) (one per warp), rows [rowt*32, rowt*32 + 32) (one
// per lane) of view v.  The spectrum table must already be in shared memory.
template <int M, bool COUNT, int MODE, bool U16>
__device__ __forceinline__ void forward_tile_of(const ForwardArgs& a, const SpecPair<M>* s_sp, IvRec* s_iv, int v,
                                             int rowt, int colb)
{
    constexpr int kSlots = iv_slots(MODE != kWalk);
    const ProjParams& P = a.p;
    const int lane = threadIdx.x;
    const int jj = colb * blockDim.y + threadIdx.y;  // detector column
    if (jj >= P.W) return;                           // whole warp exits together
    const int j = rowt * 32 + lane;                  // detector row
    const bool valid = j < P.H;
    IvRec* wbuf = s_iv + threadIdx.y * kSlots;

    const ViewGeom vg = a.views[v];
    RayPlan R;
    ray_setup(P, vg, j, jj, R);
    int Klo, Khi;
    warp_range(R, valid, Klo, Khi);

    if constexpr (COUNT) {
        SegmentCount n;
        ray_integrals<SegmentCount, M, MODE>(P, R, valid, Klo, Khi, wbuf, n, nullptr);
        const unsigned tot = __reduce_add_sync(0xffffffffu, valid ? n.nseg : 0u);
        if (lane == 0 && tot) atomicAdd(a.seg_count, (unsigned long long)tot);
        return;
    }
    float L[M];
    float* s_L = reinterpret_cast<float*>(s_iv + blockDim.y * kSlots) + threadIdx.y * 32 + lane;
    ColTab<M>* tab = nullptr;
    if (MODE == kColumns)
        tab = reinterpret_cast<ColTab<M>*>(reinterpret_cast<float*>(s_iv + blockDim.y * kSlots) +
                                           M * 32 * blockDim.y) + threadIdx.y;
    ray_path<M, MODE, U16>(a.vol, P, R, valid, Klo, Khi, wbuf, s_L, tab, L);
    if (!valid) return;
    const size_t o = ((size_t)v * P.H + (P.H - 1 - j)) * P.W + jj;
    if (a.L_out) {
#pragma unroll
        for (int i = 0; i < M; i++)
            if (i < P.nmat) a.L_out[o * P.nmat + i] = L[i];
    }
    if (a.out) {
        float I = spectral_sum<M>(s_sp, a.spec.NE, L) * R.leng;
        if (a.noise_kind != 0) {
            const uint64_t gidx = ((uint64_t)(v + a.view_offset) * P.H + (P.H - 1 - j)) * P.W + jj;
            I = (a.noise_kind == 1) ? noisy_intensity(I, a.noise_i0, a.noise_max, gidx, a.noise_seed)
                                    : poisson_intensity(I, a.noise_i0, a.noise_max, gidx, a.noise_seed);
        }
        a.out[o] = I;
    }
}

template <int M, bool COUNT, int MODE, bool U16>
__device__ __noinline__ void forward_tile_other(const ForwardArgs& a, const SpecPair<M>* s_sp, IvRec* s_iv, int v,
                                                int rowt, int colb)
{
    forward_tile_of<M, COUNT, MODE, U16>(a, s_sp, s_iv, v, rowt, colb);
}

// U16: the form the caller expects; the volume's own form decides.  The
// other one is a function of its own, so that it costs this one no registers.
template <int M, bool COUNT, int MODE, bool U16>
__device__ __forceinline__ void forward_tile(const ForwardArgs& a, const SpecPair<M>* s_sp, IvRec* s_iv, int v,
                                             int rowt, int colb)
{
    if constexpr (COUNT) forward_tile_of<M, COUNT, MODE, U16>(a, s_sp, s_iv, v, rowt, colb);
    else if (is_u16(a.vol) == U16) forward_tile_of<M, COUNT, MODE, U16>(a, s_sp, s_iv, v, rowt, colb);
    else forward_tile_other<M, COUNT, MODE, !U16>(a, s_sp, s_iv, v, rowt, colb);
}

template <int M>
__device__ __forceinline__ IvRec* iv_buffer(float4* smem, int NEmax)
{
    return reinterpret_cast<IvRec*>(reinterpret_cast<char*>(smem) + spec_bytes<M>(NEmax));
}

// Shared memory of a block: the spectral table, then per warp the interval
// buffer, the long-term sums and (col) the column table.
template <int M>
size_t block_smem(int NE, int cpb, bool sums, bool col, size_t tab = sizeof(ColTab<M>))
{
    return spec_bytes<M>(NE) + (size_t)cpb * (iv_slots(col) * sizeof(IvRec) + (sums ? M * 32 * sizeof(float) : 0) +
                                              (col ? tab : 0));
}

// grid: (ceil(W / cols_per_block), V, ceil(H / 32)); block: (32, cols_per_block).
// Blocks are dispatched view-fastest within a band of 32 detector rows, so
// the blocks resident at a time share one z band of the volume (L2 reuse
// across views).
// Register cap of the forward kernel: minimum resident 256-thread blocks per
// SM.  The walk is bound by the latency of its gathers; with one of them in
// flight behind the sums (PIPE), 4 blocks (64 registers, of which few spill: 44 to
// 84 bytes; 32 warps) are never far from the best: 448x448x120 floats, 100 x
// 100 x 60 views 1.44 ms, 5 blocks 1.40, 3 blocks 1.69, 6 without PIPE 1.55;
// 64x64x16, 32 x 32 x 60 views 0.049, 0.054, 0.045, 0.062; 64 phantoms of
// 128x128xZ, floats, flat 5.9, 5.9, 6.6 and 6.9.  The column march has more state
// and more loads in flight per warp: 3 blocks (80 registers, 24 warps) 32.1 ms
// on 512x512x200 from 360 views, 4 blocks 35.9, 2 blocks 36.6.
constexpr int fwd_min_blocks(int mode) { return mode == kWalk ? 4 : 3; }
template <int M, bool COUNT, int MODE, bool U16>
__global__ void __launch_bounds__(256, fwd_min_blocks(MODE)) forward_kernel(const __grid_constant__ ForwardArgs a)
{
    extern __shared__ float4 smem[];
    SpecPair<M>* s_sp = reinterpret_cast<SpecPair<M>*>(smem);
    load_spectrum<M>(a.spec, s_sp);
    __syncthreads();
    forward_tile<M, COUNT, MODE, U16>(a, s_sp, iv_buffer<M>(smem, a.spec.NE), blockIdx.y, a.band0 + blockIdx.z, blockIdx.x);
}

// Slices each detector row band can read, reduced over the band's rays of
// every view.  Conservative: the z cells of the ray's line over the
// iterations [klo - 1, khi] it marches (the warp-wide march reads nothing
// outside them), one cell of margin each way, and the first segment's slice.
// grid: (ceil(W / 8), V, ceil(H / 32)); block: (32, 8).
__global__ void __launch_bounds__(256) band_footprint_kernel(ProjParams P, const ViewGeom* __restrict__ views,
                                                             int* __restrict__ span)
{
    const int jj = blockIdx.x * 8 + threadIdx.y, j = blockIdx.z * 32 + threadIdx.x;
    int lo = INT_MAX, hi = -1;
    if (jj < P.W && j < P.H) {
        RayPlan R;
        ray_setup(P, views[blockIdx.y], j, jj, R);
        if (R.active) {
            if (R.first_idx >= 0) {
                const int z = R.first_idx % P.Z;
                lo = min(lo, z);
                hi = max(hi, z);
            }
            if (R.klo <= R.khi) {
                const int nzm = (int)(P.Z * 0.5);
                const double za = R.Z0 + R.Z1 * (double)(R.klo - 1), zb = R.Z0 + R.Z1 * (double)R.khi;
                const double zmin = fmin(za, zb), zmax = fmax(za, zb);
                // slice q = nzm - 1 - floor(z) (q = -1 reads slice 0)
                const double qlo = (double)(nzm - 2) - floor(zmax), qhi = (double)nzm - floor(zmin);
                if (qhi >= -1.0 && qlo <= (double)(P.Z - 1)) {
                    lo = min(lo, (int)fmax(0.0, qlo));
                    hi = max(hi, (int)fmax(0.0, fmin(qhi, (double)(P.Z - 1))));
                }
            }
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (threadIdx.x == 0 && hi >= 0) {
        atomicMin(span + 2 * blockIdx.z, lo);
        atomicMax(span + 2 * blockIdx.z + 1, hi);
    }
}

// Single-launch batched forward projection: one block per work tile of every
// item, the items' arguments in the launch's parameter block.  A block finds
// its item by a binary search over the items' first tiles; the index only
// depends on blockIdx, so the item's arguments are read from the parameter
// bank like forward_kernel's and cost no registers per thread.
template <int M, int MODE, bool U16>
__global__ void __launch_bounds__(256, fwd_min_blocks(MODE)) flat_batch_kernel(const __grid_constant__ FlatBatch b)
{
    extern __shared__ float4 smem[];
    const long long u = blockIdx.x;
    int lo = 0, hi = b.nitems - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (b.begin[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    const ForwardArgs& fa = b.fa[lo];
    SpecPair<M>* s_sp = reinterpret_cast<SpecPair<M>*>(smem);
    load_spectrum<M>(fa.spec, s_sp);
    __syncthreads();
    const long long w = u - b.begin[lo];
    const int colb = (int)(w % b.ncolb[lo]);
    const long long rest = w / b.ncolb[lo];
    const int v = (int)(rest % fa.p.V);
    const int rowt = (int)(rest / fa.p.V);
    forward_tile<M, false, MODE, U16>(fa, s_sp, iv_buffer<M>(smem, fa.spec.NE), v, rowt, colb);
}

// Tiles of a batch, taken one after another from a counter.
template <int M, class Tile>
__device__ __forceinline__ void persistent_tiles(const FlatBatch& b, unsigned long long* counter, SpecPair<M>* s_sp,
                                                 long long* s_unit, Tile tile)
{
    const long long total = b.begin[b.nitems];
    int cur = -1;
    for (;;) {
        if (threadIdx.x == 0 && threadIdx.y == 0) *s_unit = (long long)atomicAdd(counter, 1ull);
        __syncthreads();
        const long long u = *s_unit;
        if (u >= total) break;  // block-uniform
        int lo = 0, hi = b.nitems - 1;  // last item with begin <= u
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (b.begin[mid] <= u) lo = mid;
            else hi = mid - 1;
        }
        if (lo != cur) {  // block-uniform
            load_spectrum<M>(b.fa[lo].spec, s_sp);
            cur = lo;
        }
        __syncthreads();
        const long long w = u - b.begin[lo];
        const int colb = (int)(w % b.ncolb[lo]);
        const long long rest = w / b.ncolb[lo];
        const int v = (int)(rest % b.fa[lo].p.V);
        const int rowt = (int)(rest / b.fa[lo].p.V);
        tile(b.fa[lo], v, rowt, colb);
        __syncthreads();
    }
}
template <int M>
__device__ __noinline__ void persistent_tiles_any(const FlatBatch& b, unsigned long long* counter, SpecPair<M>* s_sp,
                                                  IvRec* s_iv, long long* s_unit)
{
    persistent_tiles<M>(b, counter, s_sp, s_unit, [&](const ForwardArgs& fa, int v, int rowt, int colb) {
        if (is_u16(fa.vol)) forward_tile_other<M, false, kWalk, true>(fa, s_sp, s_iv, v, rowt, colb);
        else forward_tile_other<M, false, kWalk, false>(fa, s_sp, s_iv, v, rowt, colb);
    });
}

// Persistent batched forward projection of walked items: a grid of as many
// blocks as fit on the GPU at once, every block repeatedly taking the next work
// tile from a global counter.  Tiles are numbered item by item, and within an
// item by row band, then view, then column block (the order of
// forward_kernel's grid), so the items' uneven view and slice counts
// load-balance across the whole GPU in one launch.  The items' arguments sit
// in the launch's parameter block as for flat_batch_kernel: the march reads them
// from the parameter bank (a block-uniform index found by a binary search), so
// they hold no registers; a block reloads the spectrum table only when its next
// tile belongs to another item.  The loop's state lives across the march: 5
// blocks per SM (64 phantoms of 128x128xZ 6.99 ms, 4 blocks 7.17, 6 7.54), and a
// volume of the other form (loaded since the launch was prepared) sends the
// whole loop to a function of its own, since a call within it would cost every
// tile the registers it keeps for the caller (7.32 ms).
template <int M, bool U16>
__global__ void __launch_bounds__(256, 5) persistent_batch_kernel(const __grid_constant__ FlatBatch b,
                                                                  unsigned long long* counter, int NEmax)
{
    extern __shared__ float4 smem[];
    __shared__ long long s_unit;
    SpecPair<M>* s_sp = reinterpret_cast<SpecPair<M>*>(smem);
    IvRec* s_iv = iv_buffer<M>(smem, NEmax);
    bool expected = true;
    for (int i = threadIdx.x + threadIdx.y * blockDim.x; i < b.nitems; i += blockDim.x * blockDim.y)
        expected &= is_u16(b.fa[i].vol) == U16;
    if (__syncthreads_and(expected))
        persistent_tiles<M>(b, counter, s_sp, &s_unit, [&](const ForwardArgs& fa, int v, int rowt, int colb) {
            forward_tile_of<M, false, kWalk, U16>(fa, s_sp, s_iv, v, rowt, colb);
        });
    else
        persistent_tiles_any<M>(b, counter, s_sp, s_iv, &s_unit);
}

// Register cap of the adjoint (minimum resident 256-thread blocks per SM):
// 512x512x128 floats, 45 views of 800 x 800 by shared columns, with kept path
// integrals / re-marching them: 3 blocks (80 registers) 21.9 / 40.0 ms, 4 (64) 22.8 /
// 50.2, 5 (48) 33.6 / 65.8, 2 25.3 / 43.6; 300x300x100, 40 views of 160 x 150 on
// their own: 1.71 / 3.15, 1.70 / 2.96, 1.88 / 3.02, 1.97 / 3.80.
#ifndef VCBCT_ADJ_MIN_BLOCKS
#define VCBCT_ADJ_MIN_BLOCKS 3
#endif
template <int M, bool STATE, bool COL>
__global__ void __launch_bounds__(256, VCBCT_ADJ_MIN_BLOCKS) adjoint_kernel(AdjointArgs a)
{
    extern __shared__ float4 smem[];
    constexpr int kSlots = iv_slots(COL);
    SpecPair<M>* s_sp = reinterpret_cast<SpecPair<M>*>(smem);
    IvRec* s_iv = iv_buffer<M>(smem, a.spec.NE);
    load_spectrum<M>(a.spec, s_sp);
    __syncthreads();

    const ProjParams& P = a.p;
    const int lane = threadIdx.x;
    const int colb = blockIdx.x, v = blockIdx.y, rowt = blockIdx.z;
    const int jj = colb * blockDim.y + threadIdx.y;
    if (jj >= P.W) return;
    const int j = rowt * 32 + lane;
    const bool valid = j < P.H;
    IvRec* wbuf = s_iv + threadIdx.y * kSlots;
    const ViewGeom vg = a.views[v];
    RayPlan R;
    ray_setup(P, vg, j, jj, R);
    float r = 0.0f;
    if (valid) r = a.grad_out[((size_t)v * P.H + (P.H - 1 - j)) * P.W + jj];
    const bool act = valid && r != 0.0f;
    int Klo, Khi;
    // rays with a zero residual do not scatter
    warp_range(R, act, Klo, Khi);
    if (!__any_sync(0xffffffffu, act && R.active)) return;
    // a warp none of whose segments can lie in the strip stops here (before
    // recomputing or reading its path integrals)
    const bool strip = a.y1 > a.y0;
    const bool steep = R.active && __any_sync(0xffffffffu, fabs(R.Z1) >= 1.0);
    int Klo2 = Klo, Khi2 = Khi;
    if (strip && R.active && !steep) {
        int klo = R.klo, khi = R.khi;
        strip_iterations(P, R, a.y0, a.y1, klo, khi);
        warp_range_k(klo, khi, act, Klo2, Khi2);
        const unsigned NZ = (unsigned)P.N * (unsigned)P.Z;
        const bool first_in = act && R.first_idx >= 0 &&
                              (unsigned)R.first_idx - (unsigned)a.y0 * NZ < (unsigned)(a.y1 - a.y0) * NZ;
        if (Klo2 > Khi2 && !__any_sync(0xffffffffu, first_in)) return;
    }

    // pass 1: the per-element path integrals of this ray, recomputed by a
    // first march or read from the forward projection that made them
    float L[M] = {};
    if (STATE) {
        if (act) {
            const float* Lr = a.L_in + (((size_t)v * P.H + (P.H - 1 - j)) * P.W + jj) * P.nmat;
#pragma unroll
            for (int i = 0; i < M; i++)
                if (i < P.nmat) L[i] = Lr[i];
        }
    } else {
        float* s_L = reinterpret_cast<float*>(s_iv + blockDim.y * kSlots) + threadIdx.y * 32 + lane;
        constexpr int MODE = COL ? kColumns : kWalk;
        ColTab<M>* tab = reinterpret_cast<ColTab<M>*>(reinterpret_cast<float*>(s_iv + blockDim.y * kSlots) +
                                                      M * 32 * blockDim.y) + threadIdx.y;
        if (is_u16(a.vol)) ray_path<M, MODE, true>(a.vol, P, R, act, Klo, Khi, wbuf, s_L, tab, L);
        else ray_path<M, MODE, false>(a.vol, P, R, act, Klo, Khi, wbuf, s_L, tab, L);
    }

    // d I / d L_k = -leng * sum_E pdf_E mu'_k(E) exp(-sum_k mu'_k(E) L_k)
    float g[8] = {};
    {
        f32x2 L2[M], g2[M];
#pragma unroll
        for (int k = 0; k < M; k++) {
            L2[k] = f2pack(L[k], L[k]);
            g2[k] = 0ull;
        }
        for (int e = 0; e < (a.spec.NE + 1) / 2; e++) {
            const SpecPair<M> q = s_sp[e];
            float Ta, Tb;
            f2unpack(attenuation2<M>(q, L2), Ta, Tb);
            // the hardware exponential (relative error ~1e-6, far inside the
            // gradient's 1e-5 bar): this loop runs once per ray and strip
            const f32x2 w = fmul2(q.pdf, f2pack(__expf(-Ta), __expf(-Tb)));
#pragma unroll
            for (int k = 0; k < M; k++) g2[k] = ffma2(w, q.mu[k], g2[k]);
        }
#pragma unroll
        for (int k = 0; k < M; k++) {
            float x, y;
            f2unpack(g2[k], x, y);
            g[k] = x + y;
        }
    }
    const float scale = -R.leng * r;
    const unsigned NZ = (unsigned)P.N * (unsigned)P.Z;
    Scatter<M> sc{a.grad_planes, (size_t)P.N * P.N * P.Z, P.nmat, {},
                  strip ? (unsigned)a.y0 * NZ : 0u, strip ? (unsigned)(a.y1 - a.y0) * NZ : 0xffffffffu, R.Lt};
#pragma unroll
    for (int i = 0; i < 8; i++) sc.g[i] = g[i] * scale;
    // pass 2: scatter along the same segments
    if (!R.active) return;
    if (steep) {  // the whole ray (its per-step state depends on where it starts), filtered
        if (act) {
            if (R.first_idx >= 0) sc.first(R.first_idx, R.first_len);
            if (Klo <= Khi) march(P, R, Klo, Khi, sc);
        }
        return;
    }
    if (act && R.first_idx >= 0) sc.first(R.first_idx, R.first_len);
    // only the iterations whose segments can lie in the strip's rows
    const XyPlan& xp = publish_plan<COL>(R, wbuf);
    if (Klo2 > Khi2) return;
    if (COL && (STATE || a.share)) {
        // the table takes the place of the first march's where there was one
        char* tabs = reinterpret_cast<char*>(s_iv + blockDim.y * kSlots) +
                     (STATE ? (size_t)threadIdx.y * sizeof(ScatterTab<M>)
                            : M * 32 * sizeof(float) * blockDim.y + threadIdx.y * sizeof(ColTab<M>));
        static_assert(sizeof(ScatterTab<M>) <= sizeof(ColTab<M>), "the scatter's table lies in the first march's");
        __syncwarp();
        scatter_columns<M>(P, R, xp, act, Klo2, Khi2, wbuf, reinterpret_cast<ScatterTab<M>*>(tabs), sc);
    } else {
        march_intervals(P, R, xp, act, Klo2, Khi2, wbuf, sc, []() {});
    }
}

// ------------------------------------------------------- layout kernels --
// Reference layout [Z][nmat][N][N] -> packed z-fastest records.
// grid (ceil(N/32), N, ceil(Z/32)), block (32, 8).
// A slab of nz slices [zoff, zoff + nz) of a Z-slice volume: src holds the
// slab [nz][nmat][N][N], dst the whole packed volume.
__device__ __forceinline__ void set_form(int* form, int f)
{
    if (form && blockIdx.x + blockIdx.y + blockIdx.z + threadIdx.x + threadIdx.y == 0) *form = f;
}

// 64 x by 32 z of one y: bound by memory (2 nmat bytes read and 16 written a
// voxel).  A thread reads two x of an element row at a time, all elements in
// flight, and packs their records in registers; shared memory only turns the
// order from x to z fastest, 16 bytes a lane without bank conflicts (a thread's
// two x lie 32 columns apart in it).  Where rows are 4-byte aligned the two are
// neighbours, one load (PAIR): 512x512x200 x 6 0.74 ms as floats through 2-byte
// loads, 0.34 ms now (0.22 at the copy rate).  Elsewhere they are 32 apart, so that
// either load of a warp reads one run, and neither waits behind a branch of its
// own: 203x203x77 0.069 -> 0.047 ms, 511x511x100 0.38 -> 0.25.
template <bool PAIR>
__global__ void __launch_bounds__(256) pack_u16_kernel(const uint16_t* __restrict__ src, int N, int nz, int zoff, int Z,
                                                       int nmat, uint4* __restrict__ dst, int* form)
{
    set_form(form, kFormU16);
    __shared__ uint4 tile[64][33];
    const int x0 = blockIdx.x * 64, y = blockIdx.y, z0 = blockIdx.z * 32;
    const size_t NN = (size_t)N * N;
    const int l = threadIdx.x, x = x0 + (PAIR ? 2 * l : l);
#pragma unroll 2
    for (int zz = threadIdx.y; zz < 32; zz += 8) {
        const int z = z0 + zz;
        const uint16_t* q = src + (size_t)z * nmat * NN + (size_t)y * N + x;
        const bool in = z < nz && x < N, in2 = z < nz && x + 32 < N;
        uint32_t w[8];
#pragma unroll
        for (int m = 0; m < 8; m++) {
            w[m] = 0u;
            if (PAIR) {
                if (m < nmat && in) w[m] = __ldg(reinterpret_cast<const uint32_t*>(q + m * NN));
            } else {
                const uint32_t lo = m < nmat && in ? __ldg(q + m * NN) : 0u;
                const uint32_t hi = m < nmat && in2 ? __ldg(q + m * NN + 32) : 0u;
                w[m] = lo | hi << 16;
            }
        }
        tile[l][zz] = make_uint4(__byte_perm(w[0], w[1], 0x5410), __byte_perm(w[2], w[3], 0x5410),
                                 __byte_perm(w[4], w[5], 0x5410), __byte_perm(w[6], w[7], 0x5410));
        tile[32 + l][zz] = make_uint4(__byte_perm(w[0], w[1], 0x7632), __byte_perm(w[2], w[3], 0x7632),
                                      __byte_perm(w[4], w[5], 0x7632), __byte_perm(w[6], w[7], 0x7632));
    }
    __syncthreads();
    const int z = z0 + l;
    if (z >= nz) return;
    for (int xx = threadIdx.y; xx < 64; xx += 8) {
        if (x0 + xx >= N) break;
        dst[((size_t)y * N + x0 + xx) * Z + zoff + z] = tile[PAIR ? (xx >> 1) + 32 * (xx & 1) : xx][l];
    }
}

// A thin slab (nz <= 8 slices): thread t of a 256-thread block makes record
// (y, x0 + t / 8, zoff + t % 8), so a warp writes four runs of 8 consecutive
// records and every lane has work; the tiled kernel above gives a slab of 8
// slices a quarter of its lanes.  Reads go straight to global memory (the
// block's 32 x 8 values of an element row share their sectors in L1).  grid
// (ceil(N/32), N).
__global__ void __launch_bounds__(256) pack_u16_thin_kernel(const uint16_t* __restrict__ src, int N, int nz, int zoff,
                                                            int Z, int nmat, uint4* __restrict__ dst, int* form)
{
    set_form(form, kFormU16);
    const int t = threadIdx.x;
    const int z = t & 7, x = blockIdx.x * 32 + (t >> 3), y = blockIdx.y;
    if (z >= nz || x >= N) return;
    const size_t NN = (size_t)N * N;
    const uint16_t* s = src + (size_t)z * nmat * NN + (size_t)y * N + x;
    uint32_t e[8];
#pragma unroll
    for (int m = 0; m < 8; m++) e[m] = m < nmat ? (uint32_t)__ldg(s + (size_t)m * NN) : 0u;
    dst[((size_t)y * N + x) * Z + zoff + z] =
        make_uint4(e[0] | (e[1] << 16), e[2] | (e[3] << 16), e[4] | (e[5] << 16), e[6] | (e[7] << 16));
}

// The same for float volumes, 32 x by 32 z: the record's halves are kept apart
// in shared memory and written by neighbouring lanes (whole sectors).  Bound by
// memory: 4 nmat bytes read and 32 written a voxel.  512x512x128 x 6:
// 0.62 -> 0.37 ms (0.29 at the copy rate).
__global__ void __launch_bounds__(256) pack_f32_kernel(const float* __restrict__ src, int N, int Z, int nmat,
                                                       float4* __restrict__ dst, int* form)
{
    set_form(form, kFormF32);
    // half h of column x at [h][x * 33 + z], the second 16 words on in the banks
    __shared__ float4 tile[2][32 * 33 + 4];
    const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = blockIdx.z * 32;
    const size_t NN = (size_t)N * N;
    const int l = threadIdx.x, x = x0 + l;
#pragma unroll 2
    for (int zz = threadIdx.y; zz < 32; zz += 8) {
        const int z = z0 + zz;
        float v[8];
#pragma unroll
        for (int m = 0; m < 8; m++) {
            v[m] = 0.0f;
            if (m < nmat && z < Z && x < N) v[m] = __ldg(src + ((size_t)z * nmat + m) * NN + (size_t)y * N + x);
        }
        tile[0][l * 33 + zz] = make_float4(v[0], v[1], v[2], v[3]);
        tile[1][l * 33 + zz] = make_float4(v[4], v[5], v[6], v[7]);
    }
    __syncthreads();
    for (int xx = threadIdx.y; xx < 32; xx += 8) {
        if (x0 + xx >= N) break;
        float4* col = dst + 2 * (((size_t)y * N + x0 + xx) * Z + z0);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int zz = 16 * q + (l >> 1);
            if (z0 + zz < Z) col[2 * zz + (l & 1)] = tile[l & 1][xx * 33 + zz];
        }
    }
}

// element planes [nmat][(y*N + x)*Z + z] -> [Z][nmat][N][N], accumulated (+=).
// grid (ceil(N/32), N, ceil(Z/32) * nmat), block (32, 8): a 32 x 32 (x, z)
// tile of one plane through shared memory.
__global__ void unpack_grad_kernel(const float* __restrict__ src, int N, int Z, int nmat,
                                   float* __restrict__ dst)
{
    __shared__ float tile[32][33];
    const int zt = (Z + 31) / 32;
    const int m = blockIdx.z / zt;
    const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = (blockIdx.z % zt) * 32;
    const size_t NN = (size_t)N * N;
    // element m is slot m % 4 of the group starting at element 4 (m / 4),
    // four wide, or two for a last group of one or two elements (see Scatter)
    const int e0 = (m / 4) * 4, wdt = nmat - e0 > 2 ? 4 : 2;
    const float* plane = src + (size_t)e0 * NN * Z + (m % 4);
    for (int xx = threadIdx.y; xx < 32; xx += 8) {
        const int x = x0 + xx, z = z0 + threadIdx.x;
        tile[threadIdx.x][xx] = (x < N && z < Z) ? plane[(((size_t)y * N + x) * Z + z) * wdt] : 0.0f;
    }
    __syncthreads();
    for (int zz = threadIdx.y; zz < 32; zz += 8) {
        const int z = z0 + zz, x = x0 + threadIdx.x;
        if (z >= Z || x >= N) continue;
        dst[((size_t)z * nmat + m) * NN + (size_t)y * N + x] += tile[zz][threadIdx.x];
    }
}

}  // namespace

cudaError_t launch_pack_u16(const uint16_t* src, int N, int nz, int zoff, int Z, int nmat, uint4* dst, int* form,
                            cudaStream_t st)
{
    if (nz <= 8) {
        pack_u16_thin_kernel<<<dim3((N + 31) / 32, N), 256, 0, st>>>(src, N, nz, zoff, Z, nmat, dst, form);
        return cudaGetLastError();
    }
    dim3 grid((N + 63) / 64, N, (nz + 31) / 32), block(32, 8);
    if (N % 2 == 0 && (reinterpret_cast<uintptr_t>(src) & 3) == 0)
        pack_u16_kernel<true><<<grid, block, 0, st>>>(src, N, nz, zoff, Z, nmat, dst, form);
    else
        pack_u16_kernel<false><<<grid, block, 0, st>>>(src, N, nz, zoff, Z, nmat, dst, form);
    return cudaGetLastError();
}

cudaError_t launch_pack_f32(const float* src, int N, int Z, int nmat, float4* dst, int* form, cudaStream_t st)
{
    dim3 grid((N + 31) / 32, N, (Z + 31) / 32), block(32, 8);
    pack_f32_kernel<<<grid, block, 0, st>>>(src, N, Z, nmat, dst, form);
    return cudaGetLastError();
}

cudaError_t launch_unpack_grad(const float* planes, int N, int Z, int nmat, float* dst, cudaStream_t st)
{
    dim3 grid((N + 31) / 32, N, ((Z + 31) / 32) * nmat), block(32, 8);
    unpack_grad_kernel<<<grid, block, 0, st>>>(planes, N, Z, nmat, dst);
    return cudaGetLastError();
}

template <int M, bool COUNT, int MODE, bool U16>
static cudaError_t launch_fwd_t(const ForwardArgs& a, cudaStream_t st)
{
    const int cpb = a.cols_per_block;
    dim3 block(32, cpb);
    dim3 grid((a.p.W + cpb - 1) / cpb, a.p.V, a.nbands > 0 ? a.nbands : (a.p.H + 31) / 32);
    const size_t shm = block_smem<M>(a.spec.NE, cpb, true, MODE != kWalk);
    auto k = forward_kernel<M, COUNT, MODE, U16>;
    const cudaError_t e = allow_smem(k, shm);
    if (e != cudaSuccess) return e;
    k<<<grid, block, shm, st>>>(a);
    return cudaGetLastError();
}

// The kernels and the shared memory of a launch of batch items of one kind.
struct BatchKernels {
    void (*persistent)(FlatBatch, unsigned long long*, int);  // walked items only
    void (*flat)(FlatBatch);
    size_t shm;
};
template <int M, int MODE, bool U16>
static BatchKernels batch_kernels_of(const BatchShape& s)
{
    BatchKernels k{nullptr, flat_batch_kernel<M, MODE, U16>, block_smem<M>(s.NEmax, s.cols_per_block, true, MODE != kWalk)};
    if constexpr (MODE == kWalk) k.persistent = persistent_batch_kernel<M, U16>;
    return k;
}
template <int M>
static BatchKernels batch_kernels_of(const BatchShape& s)
{
    if (s.columns) return s.u16 ? batch_kernels_of<M, kColumns, true>(s) : batch_kernels_of<M, kColumns, false>(s);
    return s.u16 ? batch_kernels_of<M, kWalk, true>(s) : batch_kernels_of<M, kWalk, false>(s);
}
static BatchKernels batch_kernels(const BatchShape& s)
{
    return s.nmat_max <= 6 ? batch_kernels_of<6>(s) : batch_kernels_of<8>(s);
}

cudaError_t launch_persistent_batch(const FlatBatch& b, const BatchShape& s, int blocks, unsigned long long* counter,
                                    cudaStream_t st)
{
    if (b.begin[b.nitems] <= 0) return cudaSuccess;
    dim3 block(32, s.cols_per_block);
    // (the shared-memory attribute is set by batch_blocks_per_sm, before any
    // stream capture)
    cudaError_t e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    const BatchKernels k = batch_kernels(s);
    k.persistent<<<blocks, block, k.shm, st>>>(b, counter, s.NEmax);
    return cudaGetLastError();
}

cudaError_t launch_flat_batch(const FlatBatch& b, const BatchShape& s, cudaStream_t st)
{
    const long long total = b.begin[b.nitems];
    if (total <= 0) return cudaSuccess;
    if (total > 0x7fffffffLL) return cudaErrorInvalidValue;
    dim3 block(32, s.cols_per_block);
    const BatchKernels k = batch_kernels(s);
    // (the shared-memory attribute is set by batch_blocks_per_sm, before any
    // stream capture)
    k.flat<<<(unsigned)total, block, k.shm, st>>>(b);
    return cudaGetLastError();
}

int batch_blocks_per_sm(const BatchShape& s)
{
    const BatchKernels k = batch_kernels(s);
    int n = 0;
    // (the persistent kernel holds its tile's number in static shared memory)
    if (allow_smem(k.flat, k.shm) != cudaSuccess || !k.persistent ||
        allow_smem(k.persistent, k.shm, kSmemMost - 1024) != cudaSuccess)
        return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k.persistent, 32 * s.cols_per_block, k.shm);
    return n;
}

cudaError_t launch_band_footprint(const ProjParams& P, const ViewGeom* d_views, int* d_span, cudaStream_t st)
{
    dim3 grid((P.W + 7) / 8, P.V, (P.H + 31) / 32), block(32, 8);
    band_footprint_kernel<<<grid, block, 0, st>>>(P, d_views, d_span);
    return cudaGetLastError();
}

// What the rules for shared columns look at.
struct ColumnShape {
    double rays;    // of a detector column per slice at the isocentre
    double planes;  // z planes that the detector's steepest ray meets in a batch of steps
    double inside;  // the same of the steepest ray that stays in the slab, a little less where many rays leave it
    double slices;  // that a warp's rays meet at the far end of the cylinder
    bool whole;     // 1 / s is an integer: no dominant-axis plane lies inside a step
    bool small;     // below 2e6 voxels: gathers hit L1 and L2
};
static ColumnShape column_shape(const ProjParams& p)
{
    ColumnShape c;
    const double pitch = p.piso * p.dpn / p.H, half = p.piso * p.dpn / 2.0;
    const double per_batch = 32.0 * p.s / p.sad / p.step;
    c.rays = p.step / pitch;
    c.planes = per_batch * half;
    const double in_slab = fmin(1.0, p.Z * p.step / 2.0 / half);
    c.inside = c.planes * in_slab * sqrt(sqrt(in_slab));
    c.slices = 32.0 * pitch * (1.0 + p.N * p.s / 2.0 / p.sad) / p.step + c.planes + 1.0;
    c.whole = fabs(1.0 / p.s - rint(1.0 / p.s)) < 1e-6;
    c.small = (double)p.N * p.N * p.Z < 2e6;
    return c;
}

// Enough rays to a slice.  Columns against the walk on B200, times uint16 /
// float: at 1.15 rays 1.6 / 1.2 (448x448x120) and 1.15-1.2 / 0.94-0.99
// (256x256x64), at 0.95 0.9-1.15 / 0.8-0.98 everywhere, at 3.1 2.2 / 1.8.  Small
// volumes also ask that a warp's rays meet no more than 32 slices (batches of steps
// beyond that fall back to a walk, which small volumes do not repay) unless
// those inside the slab meet few planes.  Columns / walk, uint16 (float), at 1.15
// rays and 34-37 slices: 1.31 (1.16) at 0.45 planes (128x128x14), 1.15 (1.03) at
// 0.83 (128x128x26), 0.87 (0.79) at 1.66 (128x128x52); where 1 / s is not an
// integer 1.39 (1.30) at 0.6 (96x96x14), 1.16 (1.06) at 1.54 (96x96x36), 0.89 (0.81)
// at 2.05 (96x96x48).
static bool rays_share_slices(const ColumnShape& c)
{
    return c.rays >= 1.15 && (!c.small || c.slices <= 32.8 || c.inside <= (c.whole ? 0.9 : 1.6));
}

bool march_shares_columns(const ProjParams& p)
{
    // One line for both forms, whose projections agree bit for bit.  A ray's
    // chunk with a z plane in it costs more here than in the walk, so the more
    // planes the rays inside the slab meet, the more of them have to share a slice;
    // the walk pays more for a plane itself where its intervals hold
    // dominant-axis planes too (1 / s not an integer) or its gathers miss the
    // caches.  B200, float columns, float walk (uint16 columns, uint16 walk), each
    // against the walk as it was before there were columns, 60 views of 64 columns:
    //   whole, 1.15 planes: 0.95, 0.94 (0.85, 1.00) at 1.5 rays (128x128x36)
    //   whole, 1.54: 1.07, 0.96 (0.97, 1.01) at 1.3, 0.97, 0.92 (0.85, 0.98) at 1.8 (128x128x48)
    //   whole, 1.54: 0.98, 0.93 (0.81, 0.93) at 1.3 (256x256x96)
    //   whole, 1.92: 1.15, 0.93 (1.02, 0.95) at 1.3, 1.00, 0.96 (0.87, 1.02) at 1.8 (256x256x120)
    //   whole, 2.30: 1.10, 0.92 (1.00, 1.00) at 1.8, 0.94, 0.90 (0.85, 0.99) at 2.8 (128x128x72)
    //   whole, 2.56: 1.14, 0.96 (1.01, 1.02) at 1.8, 1.04, 0.98 (0.92, 1.09) at 2.8 (256x256x160)
    //   whole, 3.07: 1.12, 0.92 (1.03, 1.03) at 2.2, 1.00, 0.91 (0.90, 1.04) at 3.6 (128x128x96)
    //   not, 1.84: 0.95, 0.91 (0.87, 0.99) at 1.3 (160x160x72)
    //   not, 1.94: 0.72, 0.92 (0.68, 1.01) at 1.3 (203x203x96)
    //   not, 2.46: 1.07, 0.94 (0.96, 1.05) at 1.8, 0.98, 0.93 (0.89, 1.05) at 2.2 (160x160x96)
    //   not, 3.07: 1.08, 0.92 (1.00, 0.96) at 1.8, 0.96, 0.88 (0.89, 0.97) at 2.2 (64x64x48)
    const ColumnShape c = column_shape(p);
    const double least = !c.whole  ? fmin(2.2, 1.15 + 1.5 * (c.inside - 2.0))
                         : c.small ? 1.15 + 1.35 * (c.inside - 1.3)
                                   : fmin(2.6, 1.15 + 2.5 * (c.inside - 1.5));
    return rays_share_slices(c) && c.rays >= least;
}

bool scatter_shares_columns(const ProjParams& p)
{
    // The scatter's own line: a ray's walk of the chunks in which it meets a z
    // plane costs more than the forward's, so it also asks that the steepest
    // ray meet few of them per batch of steps, and the more of them the rays
    // inside the slab meet, the more rays to a slice.  B200, times by shared columns /
    // walked: 1.66 at 3.1 rays and 2.1 planes (512x512x128, 45 views of 800 x 800), 0.9
    // at 1.3 and 5.8 (74x74x39), 0.7 at 1.4 and 3.7 (146x146x140); by the planes
    // inside the slab, large volumes 1.08 at 1.0 and 1.45 rays (256x256x65), 0.84 at
    // 2.0 and 1.45, 0.92 and 1.8, 1.07 and 2.4 (215x215x110), small ones 0.98 at 0.7
    // and 1.45, 1.15 and 1.8 (128x128x26), 0.85 at 1.8 and 1.8, 0.97 and 2.4, 1.08
    // and 3.5 (96x96x44).
    const ColumnShape c = column_shape(p);
    const double least = fmax(1.4, c.small ? 1.7 + 0.9 * (c.inside - 0.8) : 1.4 + 0.75 * (c.inside - 1.2));
    return rays_share_slices(c) && c.planes <= 2.5 && c.rays >= least;
}

cudaError_t launch_forward(const ForwardArgs& a, cudaStream_t st)
{
    if (a.seg_count) return launch_fwd_t<6, true, kWalk, false>(a, st);
    const bool u16 = a.vol.expect == kFormU16;
    auto launch = [&](auto m, auto u) {
        constexpr int M = decltype(m)::value;
        constexpr bool U = decltype(u)::value;
        if (a.columns) return launch_fwd_t<M, false, kColumns, U>(a, st);
        return launch_fwd_t<M, false, kWalk, U>(a, st);
    };
    using std::integral_constant;
    if (a.p.nmat <= 6)
        return u16 ? launch(integral_constant<int, 6>{}, std::true_type{}) : launch(integral_constant<int, 6>{}, std::false_type{});
    return u16 ? launch(integral_constant<int, 8>{}, std::true_type{}) : launch(integral_constant<int, 8>{}, std::false_type{});
}

template <int M, bool STATE, bool COL>
static cudaError_t launch_adj_t(const AdjointArgs& a, cudaStream_t st)
{
    const int cpb = a.cols_per_block;
    dim3 block(32, cpb);
    // the forward's block order; (columns, row bands, views) and (views,
    // columns, row bands) measured within 3 % on B200
    dim3 grid((a.p.W + cpb - 1) / cpb, a.p.V, (a.p.H + 31) / 32);
    const size_t shm = block_smem<M>(a.spec.NE, cpb, !STATE, COL, STATE ? sizeof(ScatterTab<M>) : sizeof(ColTab<M>));
    auto k = adjoint_kernel<M, STATE, COL>;
    const cudaError_t e = allow_smem(k, shm);
    if (e != cudaSuccess) return e;
    k<<<grid, block, shm, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint(const AdjointArgs& a, cudaStream_t st)
{
    using std::integral_constant;
    auto launch = [&](auto m, auto col) {
        constexpr int M = decltype(m)::value;
        constexpr bool COL = decltype(col)::value;
        return a.L_in ? launch_adj_t<M, true, COL>(a, st) : launch_adj_t<M, false, COL>(a, st);
    };
    const bool col = a.L_in ? a.share : a.columns;
    if (a.p.nmat <= 6)
        return col ? launch(integral_constant<int, 6>{}, std::true_type{}) : launch(integral_constant<int, 6>{}, std::false_type{});
    return col ? launch(integral_constant<int, 8>{}, std::true_type{}) : launch(integral_constant<int, 8>{}, std::false_type{});
}

}  // namespace vcbct
