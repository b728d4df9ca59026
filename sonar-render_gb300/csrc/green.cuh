// green.cuh -- the FP32 pair arithmetic shared by the kernels that evaluate
// single FACET_SELF entries: the reference's rounded dot product and cosine
// gate (src/OptiX.cu:267-330) and the entry T(j, i) of the low-rank blocks
// (the Green's function of the symmetric bounce sum, src/OptiX.cu:340-390).
#pragma once

#include "sonar_internal.h"

namespace sonar {
namespace {

constexpr float kInv4Pi = 0.0795774715459476679f;  // 1 / (4 pi)
constexpr float kTwoPi = 6.28318530717958647692f;

__device__ __forceinline__ float dot_rn(float ax, float ay, float az, float bx, float by, float bz)
{
    // a.x*b.x + a.y*b.y + a.z*b.z evaluated left to right, every product and
    // sum rounded separately (the reference's vec_math dot without contraction)
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// Cosine gates.  The reference's decision is "cos < 1e-6 -> skip" with
// cos = dot(v * (1/r), n) in FP32 without contraction (exact_cos below).  A
// cheaper estimate dot(v, n) * rsqrt(v.v) differs from it by less than 7e-7
// (both are within a few ulp of the true cosine, |cos| <= 1), so outside the
// band [0, 2e-6] the estimate decides the same way; inside it the exact
// expression is evaluated.
__device__ __forceinline__ float exact_cos(float vx, float vy, float vz, float sign, float nx, float ny, float nz)
{
    const float r = __fsqrt_rn(dot_rn(vx, vy, vz, vx, vy, vz));
    const float inv = __frcp_rn(r);
    const float ux = __fmul_rn(vx, inv), uy = __fmul_rn(vy, inv), uz = __fmul_rn(vz, inv);
    return dot_rn(sign * ux, sign * uy, sign * uz, nx, ny, nz);
}

// The exact FP32 cosine gate where the estimate is inside the band (rare):
// kept out of line so that kernels that unroll several entries carry one
// copy of it.
__device__ __noinline__ bool gate_exact(float vx, float vy, float vz, float sign, float nx, float ny, float nz)
{
    return !(exact_cos(vx, vy, vz, sign, nx, ny, nz) < 1e-6f);
}

__device__ __forceinline__ bool gate_est(float est, float vx, float vy, float vz, float sign, float nx, float ny,
                                         float nz)
{
    if (est > 2e-6f) return true;
    if (est < 0.0f) return false;
    return gate_exact(vx, vy, vz, sign, nx, ny, nz);
}

// T(j, i) of one pair of a block of class cls (bit: the pair's mask bit for
// BITS; CLEAR blocks evaluate the cosine gates inline).  One code path for
// every class: the Green's function of sym_pair (same operations, same
// rounding), then the pair's gate.
template <bool ATT>
__device__ __forceinline__ float2 lr_entry(const SumArgs &a, int cls, bool bit, float4 pi, float4 ni, float4 pj,
                                           float4 nj)
{
    const float vx = __fsub_rn(pj.x, pi.x), vy = __fsub_rn(pj.y, pi.y), vz = __fsub_rn(pj.z, pi.z);
    const float r2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
    const float rinv = rsqrtf(r2);
    const float r0 = r2 * rinv;
    const float r = fmaf(fmaf(-r0, r0, r2), 0.5f * rinv, r0);
    const float th = __fmul_rn(r, a.k2hi);
    const float tl = fmaf(r, a.k2lo, fmaf(r, a.k2hi, -th));
    const float frac = (th - rintf(th)) + tl;
    float sn, cs;
    __sincosf(frac * kTwoPi, &sn, &cs);
    const float d1 = vx * ni.x + vy * ni.y + vz * ni.z;  // r cos_scat
    const float d2 = vx * nj.x + vy * nj.y + vz * nj.z;  // -r cos_inc
    const float rinv2 = rinv * rinv;
    const float u = (d1 * d2) * (-rinv2);
    float Tr, Ti;
    if (ATT) {
        const float amp = rinv * kInv4Pi * __expf(-a.ka * r);
        Tr = u * fmaf(amp, fmaf(a.ka, cs, a.kr * sn), rinv2);
        Ti = u * (amp * fmaf(a.ka, sn, -a.kr * cs));
    } else {
        const float ua = (u * rinv) * a.kr4pi;
        Tr = fmaf(ua, sn, u * rinv2);
        Ti = -ua * cs;
    }
    float rr = r;
    if (fabsf(r - a.rmin) <= a.rmin * 1e-6f) rr = __fsqrt_rn(dot_rn(vx, vy, vz, vx, vy, vz));
    if (rr < a.rmin) {
        Tr = u * (-a.ka * kInv4Pi);
        Ti = u * (a.kr * kInv4Pi);
    }
    bool ok = cls == kFlagBits ? bit : true;
    if (cls == kFlagClear)
        ok = gate_est(d1 * rinv, vx, vy, vz, 1.0f, ni.x, ni.y, ni.z) &&
             gate_est(-d2 * rinv, vx, vy, vz, -1.0f, nj.x, nj.y, nj.z);
    return ok ? make_float2(Tr, Ti) : make_float2(0.0f, 0.0f);
}

struct Dst {
    float px, py, pz;
    float nx, ny, nz;
};

// Gate from an estimate already at hand (same band rule as cos_gate): the
// decision always equals the reference's exact FP32 one.
__device__ __forceinline__ bool gate_from(float est, float vx, float vy, float vz, float sign, float nx, float ny,
                                          float nz)
{
    if (est > 2e-6f) return true;
    if (est < 0.0f) return false;
    return !(exact_cos(vx, vy, vz, sign, nx, ny, nz) < 1e-6f);
}

// T_ij = cos_scat cos_inc G of one FACET_SELF pair (weights excluded; the
// symmetric bounce sum's arithmetic).  GATE: the pair's cosine gates in ok;
// REG: the regularised branch.
template <bool ATT, bool GATE, bool REG>
__device__ __forceinline__ void sym_pair(const SumArgs &a, const float4 A, const float4 B, const Dst &d, float &Tr,
                                         float &Ti, bool &ok)
{
    const float vx = __fsub_rn(d.px, A.x), vy = __fsub_rn(d.py, A.y), vz = __fsub_rn(d.pz, A.z);
    // |v|^2 with fused multiply-adds; r from one Newton step on rsqrt (within an
    // ulp or two of the reference's FP32 r; the regularisation branch below
    // recomputes the reference's r exactly where it decides)
    const float r2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
    const float rinv = rsqrtf(r2);
    const float r0 = r2 * rinv;
    const float r = fmaf(fmaf(-r0, r0, r2), 0.5f * rinv, r0);
    const float th = __fmul_rn(r, a.k2hi);
    const float tl = fmaf(r, a.k2lo, fmaf(r, a.k2hi, -th));
    const float frac = (th - rintf(th)) + tl;
    float sn, cs;
    __sincosf(frac * kTwoPi, &sn, &cs);
    const float d1 = vx * B.x + vy * B.y + vz * B.z;    // r cos_scat (source side)
    const float d2 = vx * d.nx + vy * d.ny + vz * d.nz;  // -r cos_inc (destination side)
    ok = true;
    if (GATE)
        ok = gate_from(d1 * rinv, vx, vy, vz, 1.0f, B.x, B.y, B.z) &&
             gate_from(-d2 * rinv, vx, vy, vz, -1.0f, d.nx, d.ny, d.nz);
    // T = cos_scat cos_inc G,  G = -e^{ikr}/(4 pi) (ik/r) + 1/r^2
    const float rinv2 = rinv * rinv;
    const float u = (d1 * d2) * (-rinv2);  // cos_scat cos_inc
    if (ATT) {
        const float amp = rinv * kInv4Pi * __expf(-a.ka * r);
        Tr = u * fmaf(amp, fmaf(a.ka, cs, a.kr * sn), rinv2);
        Ti = u * (amp * fmaf(a.ka, sn, -a.kr * cs));
    } else {
        const float ua = (u * rinv) * a.kr4pi;
        Tr = fmaf(ua, sn, u * rinv2);
        Ti = -ua * cs;
    }
    if (REG) {
        // regularised G below r_min = delta_src (OptiX.cu:340-346), decided with
        // the reference's r where it is close to the threshold
        float rr = r;
        if (fabsf(r - a.rmin) <= a.rmin * 1e-6f) rr = __fsqrt_rn(dot_rn(vx, vy, vz, vx, vy, vz));
        if (rr < a.rmin) {
            Tr = u * (-a.ka * kInv4Pi);
            Ti = u * (a.kr * kInv4Pi);
        }
    }
}

// order-preserving float <-> int map for shared-memory atomic min / max
__device__ __forceinline__ int f2o(float f)
{
    const int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// minimum distance between two axis-aligned boxes
__device__ __forceinline__ float box_gap(float4 lo1, float4 hi1, float4 lo2, float4 hi2)
{
    const float gx = fmaxf(0.0f, fmaxf(lo1.x - hi2.x, lo2.x - hi1.x));
    const float gy = fmaxf(0.0f, fmaxf(lo1.y - hi2.y, lo2.y - hi1.y));
    const float gz = fmaxf(0.0f, fmaxf(lo1.z - hi2.z, lo2.z - hi1.z));
    return sqrtf(fmaf(gx, gx, fmaf(gy, gy, gz * gz)));
}

// upper bound of the distance between points of two boxes
__device__ __forceinline__ float box_diag(float4 lo1, float4 hi1, float4 lo2, float4 hi2)
{
    return fmaxf(hi1.x, hi2.x) - fminf(lo1.x, lo2.x) + (fmaxf(hi1.y, hi2.y) - fminf(lo1.y, lo2.y)) +
           (fmaxf(hi1.z, hi2.z) - fminf(lo1.z, lo2.z));
}

// largest |coordinate| of a box
__device__ __forceinline__ float box_extent(float4 lo, float4 hi)
{
    return fmaxf(fmaxf(fmaxf(fabsf(lo.x), fabsf(lo.y)), fmaxf(fabsf(lo.z), fabsf(hi.x))), fmaxf(fabsf(hi.y), fabsf(hi.z)));
}

// Do the intermediate values of the packed forms stay within FP32 for pairs
// between gap and diag apart and weights up to w?  They leave k / (4 pi), and
// on one-facet tiles the plane distances, to the end of a tile's sum, so their
// terms can be larger than the sum by 4 pi / (k r^2); the scalar form, which
// meets none of them, takes the rest (and weights that are not finite).
// 512: the terms of 256 complex products.
__device__ __forceinline__ bool packed_in_range(const SumArgs &a, float gap, float diag, float w)
{
    const float g = 1.0f / gap;
    const float grow = a.ka < 0.0f ? __expf(-a.ka * diag) : 1.0f;
    const float t = g * g * fmaxf(g, 1.0f) * (g / a.kr4pi + 1.0f + fabsf(a.ka / a.kr)) * grow;
    return t * fmaxf(1.0f, 512.0f * w * fmaxf(1.0f, diag)) < 1e37f;
}

// Error-free sum of two FP32 values (Knuth's two-sum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// n.p - (chi + clo), the products and sums carried in two FP32 words: the
// distance of a point from a tile's plane without the cancellation of a
// single-word evaluation.
__device__ __forceinline__ float plane_distance(const TileGeom &g, float x, float y, float z)
{
    const float hx = g.n.x * x, hy = g.n.y * y, hz = g.n.z * z;
    float l = fmaf(g.n.x, x, -hx) + fmaf(g.n.y, y, -hy) + fmaf(g.n.z, z, -hz);
    float s, e;
    two_sum(hx, hy, s, e);
    l += e;
    two_sum(s, hz, s, e);
    l += e;
    two_sum(s, -g.lo.w, s, e);
    l += e;
    return s + (l - g.hi.w);
}

}  // namespace
}  // namespace sonar
