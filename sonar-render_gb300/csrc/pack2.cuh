// pack2.cuh -- two FP32 values per register pair: the packed multiply-add
// forms of sm_100 and later (fma/mul/add/sub .rn.f32x2, each half rounded
// exactly like the scalar operation) and the phase reduction the packed pair
// loops share.
//
// Why packed: the pair sums are bound by instruction issue (about 57
// instructions per unordered pair against one warp instruction per clock and
// scheduler).  A packed operation does two pairs' arithmetic in one issue
// slot; the FP32 lanes and the special-function unit, which set the floor,
// are then the only limits left.
#pragma once

#include <cuda_runtime.h>

namespace sonar {
namespace {

using f2 = unsigned long long;  // two FP32 values, low half first

__device__ __forceinline__ f2 pk2(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2 dup2(float v) { return pk2(v, v); }
__device__ __forceinline__ void up2(f2 v, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float sum2(f2 v)
{
    float a, b;
    up2(v, a, b);
    return a + b;
}

// v.v of two vectors with every product and sum rounded by itself (the
// reference's vec_math dot).  The sums are scalar: the assembler contracts a
// packed product and a packed sum into one fused operation, whatever their
// rounding modifiers say (measured: a quarter of random operands differ).
__device__ __forceinline__ f2 dot_rn2(f2 vx, f2 vy, f2 vz)
{
    float x0, x1, y0, y1, z0, z1;
    up2(mul2(vx, vx), x0, x1);
    up2(mul2(vy, vy), y0, y1);
    up2(mul2(vz, vz), z0, z1);
    return pk2(__fadd_rn(__fadd_rn(x0, y0), z0), __fadd_rn(__fadd_rn(x1, y1), z1));
}

// 1 / sqrt of a normal positive number (callers exclude denormals: no scaling code)
__device__ __forceinline__ float rsqrt_fast(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ f2 rsqrt2(f2 x)
{
    float a, b;
    up2(x, a, b);
    return pk2(rsqrt_fast(a), rsqrt_fast(b));
}
__device__ __forceinline__ f2 rcp2(f2 x)
{
    float a, b, ra, rb;
    up2(x, a, b);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(a));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(b));
    return pk2(ra, rb);
}
// two register pairs of a 16-byte shared-memory word
__device__ __forceinline__ ulonglong2 ld2(const float4 *p) { return *reinterpret_cast<const ulonglong2 *>(p); }
// the halves whose bit of m is set, 0 for the others
__device__ __forceinline__ f2 pick2(f2 v, unsigned m)
{
    float a, b;
    up2(v, a, b);
    return pk2((m & 1u) ? a : 0.0f, (m & 2u) ? b : 0.0f);
}
__device__ __forceinline__ f2 ex2_2(f2 x)
{
    float a, b, ea, eb;
    up2(x, a, b);
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ea) : "f"(a));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(eb) : "f"(b));
    return pk2(ea, eb);
}

// Adding and subtracting 1.5 * 2^23 rounds to an integer (round to nearest
// even, any integer of at most a few units off beyond 2^22, which the phase
// does not see) on the multiply-add pipe; rintf runs on the special-function
// unit, which the sine, cosine and square root already fill.
constexpr float kRoundMagic = 12582912.0f;

// Constants of the phase in turns, k r / (2 pi) = r (khi + klo).
struct Phase2 {
    f2 khi, klo, nhalf_khi, magic, neg1, two_pi;
};
__device__ __forceinline__ Phase2 phase2(float k2hi, float k2lo)
{
    return Phase2{dup2(k2hi), dup2(k2lo), dup2(-0.5f * k2hi), dup2(kRoundMagic), dup2(-1.0f),
                  dup2(6.28318530717958647692f)};
}

// sine and cosine of f turns (|f| about 1/2 at most)
__device__ __forceinline__ void turns_sincos2(const Phase2 &p, f2 f, f2 &sn, f2 &cs)
{
    float a, b, s0, c0, s1, c1;
    up2(mul2(f, p.two_pi), a, b);
    __sincosf(a, &s0, &c0);
    __sincosf(b, &s1, &c1);
    sn = pk2(s0, s1);
    cs = pk2(c0, c1);
}

// sine and cosine of k r, r = r0 + c with r0 = fl(r2 rinv) and the Newton
// correction c = -r0 (r0 rinv - 1) / 2 (half an ulp of r0 at most once
// added).  Turns: the integer part q = round(r0 khi) comes out of one fused
// multiply-add with the rounding constant; r0 khi - q is exact to 2^-26 in
// one fused step, and r0 klo and c khi are added to that small number, so r
// itself is never rounded to FP32.
__device__ __forceinline__ void sincos2(const Phase2 &p, f2 r0, f2 rinv, f2 &sn, f2 &cs)
{
    const f2 e = fma2(fma2(r0, rinv, p.neg1), p.nhalf_khi, p.klo);
    const f2 m = fma2(r0, p.khi, p.magic);
    const f2 nq = sub2(p.magic, m);
    const f2 f = fma2(r0, p.khi, nq);
    turns_sincos2(p, fma2(r0, e, f), sn, cs);
}

}  // namespace
}  // namespace sonar
