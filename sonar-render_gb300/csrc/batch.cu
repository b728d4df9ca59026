// batch.cu -- many sources, receivers, frequencies and scenes in one launch.
//
// The reference answers "what does receiver p hear when source q radiates"
// one source at a time: load_source_points({q}), ProjectSrcPointsToObjects
// (source -> every fragment cell, src/OptiX.cu:35-110) and
// ProjectTargetToFieldPoints (every fragment -> every field point,
// src/OptiX.cu:112-190).  For S sources and R receivers over N fragments
// that is S * (N + N * R) Green's function evaluations, and the readout
// kernel G(p, n) = A_n cos_scat(n -> p) G(r_pn) is recomputed for every
// source although it does not depend on it.
//
// Here the two hops of one (scene, frequency) item become one complex
// matrix product
//     out[p][q] = sum_n  G(p, n) * Pinc(n, q),
//     Pinc(n, q) = cos_inc(q -> n) e^{ikr}/r  (unit source pressure),
// with both factors materialised tile by tile in shared memory (R + S
// evaluations per fragment instead of S (1 + R)) and contracted on the
// tensor cores:
//   * complex -> real: D (128 x 64) = [[Gr, -Gi], [Gi, Gr]] (128 x 2K) times
//     [Pr; Pi] (2K x 64): rows 0..63 of D are Re out, rows 64..127 Im out;
//   * split BF16: every FP32 value x = hi + lo with hi = bf16(x),
//     lo = bf16(x - hi); D += Ahi Bhi + Ahi Blo + Alo Bhi (relative error of
//     a product about 2^-16), accumulated in FP32 in tensor memory;
//   * tcgen05.mma (kind::f16, M = 128, N = 64, K = 16) issued by one thread,
//     operands in the no-swizzle K-major canonical layout (8-row x 16-byte
//     core matrices), completion tracked by tcgen05.commit on an mbarrier per
//     operand stage (two stages: the next tile is generated while the tensor
//     core consumes the previous one);
//   * the accumulator is read back with tcgen05.ld at the end of each
//     segment (at most kBatchSegChunks chunks, so that an FP32 accumulation
//     never spans more than a few thousand fragments) into FP32 partials
//     that k_batch_reduce adds per item in a fixed order (compensated
//     FP32 summation, the head and tail combined in FP64).
// One persistent launch covers every chunk of every item: CTA b processes a
// contiguous range of the global chunk list (balanced over the grid), cut
// into segments at item boundaries.
//
// Visibility: per fragment one 64-bit word per hop (k_batch_vis: the cosine
// gates and the shadow test of every pair) gates the entries.
#include "sonar_internal.h"
#include "tc05.cuh"
#include "pack2.cuh"

#include <cstdint>

namespace sonar {
namespace {

constexpr int kBatchThreads = 256;
constexpr uint32_t kTmemCols = 64;          // FP32 accumulator: 128 lanes x 64 columns
constexpr int kGenGroup = 2;                // fragment pairs whose entries are evaluated together

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N = 64, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 3) << 17) |
                            ((uint32_t)(128 >> 4) << 24);

// ---------------------------------------------------------------- the two kernels of an item
// Both entries are evaluated for two fragments at a time, a fragment to each
// half of a register pair (pack2.cuh): the scalar form took 8.6e8 warp
// instructions for 3.97 M fragments x 128 points, this one 5.8e8.  What bounds
// it now is the wait at the chunk's barrier and the chains of its few warps (16
// an SM, by shared memory).  1.56 -> 1.16 ms; groups of one pair 1.28, of four
// 1.17.  Constants of the current item:
struct Gen2 {
    Phase2 ph;
    f2 half, c4pik, natt, qatt, nqatt;
};
__device__ __forceinline__ Gen2 gen2(const BatchItem &it)
{
    const float q = it.ka / it.kr;
    return Gen2{phase2(it.k2hi, it.k2lo), dup2(0.5f),  dup2(1.0f / it.kr4pi), dup2(-it.ka * 1.44269504088896341f),
                dup2(q),                  dup2(-q)};
}

// sine and cosine of k r with r rounded like the reference's distance (|v|^2
// without contraction, r within an ulp of the rounded root)
__device__ __forceinline__ void wave2(const Gen2 &g, f2 r2, f2 rinv, f2 &r, f2 &sn, f2 &cs)
{
    const f2 r0 = mul2(r2, rinv);
    r = fma2(fma2(r0 ^ 0x8000000080000000ull, r0, r2), mul2(rinv, g.half), r0);
    const f2 f = fma2(r, g.ph.khi, sub2(g.ph.magic, fma2(r, g.ph.khi, g.ph.magic)));
    turns_sincos2(g.ph, fma2(r, g.ph.klo, f), sn, cs);
}

// Readout entries G(p, n) = A_n cos_scat G(r), G = -e^{ikr}/(4 pi) (ik/r) + 1/r^2
// (src/OptiX.cu:150-186; cos_scat from the fragment's facet normal), as
// (Gr, -Gi).  F: the pair's staged data, its areas times k / (4 pi).
template <bool ATT>
__device__ __forceinline__ void readout2(const Gen2 &g, const float4 *F, f2 px, f2 py, f2 pz, f2 &gr, f2 &ngi)
{
    const ulonglong2 XY = ld2(F), ZA = ld2(F + 1), NXY = ld2(F + 4), NZ = ld2(F + 5);
    const f2 vx = sub2(px, XY.x), vy = sub2(py, XY.y), vz = sub2(pz, ZA.x);
    const f2 r2 = dot_rn2(vx, vy, vz), rinv = rsqrt2(r2);
    f2 r, sn, cs;
    wave2(g, r2, rinv, r, sn, cs);
    const f2 d = fma2(vx, NXY.x, fma2(vy, NXY.y, mul2(vz, NZ.x)));  // r cos_scat
    const f2 w = mul2(mul2(mul2(rinv, rinv), d), ZA.y);
    if (ATT) {
        const f2 osc = mul2(w, ex2_2(mul2(r, g.natt)));
        gr = fma2(osc, fma2(g.qatt, cs, sn), mul2(w, mul2(rinv, g.c4pik)));
        ngi = mul2(osc, fma2(g.nqatt, sn, cs));
    } else {
        gr = mul2(w, fma2(rinv, g.c4pik, sn));
        ngi = mul2(w, cs);
    }
}

// Incident entries Pinc(n, q) = cos_inc e^{ikr} / r at the fragments'
// source-hop centroids (src/OptiX.cu:45-106; unit source pressure).
template <bool ATT>
__device__ __forceinline__ void incident2(const Gen2 &g, const float4 *F, f2 qx, f2 qy, f2 qz, f2 &pr, f2 &pi)
{
    const ulonglong2 XY = ld2(F + 2), ZW = ld2(F + 3), NXY = ld2(F + 4), NZ = ld2(F + 5);
    const f2 vx = sub2(qx, XY.x), vy = sub2(qy, XY.y), vz = sub2(qz, ZW.x);
    const f2 r2 = dot_rn2(vx, vy, vz), rinv = rsqrt2(r2);
    f2 r, sn, cs;
    wave2(g, r2, rinv, r, sn, cs);
    f2 amp = mul2(fma2(vx, NXY.x, fma2(vy, NXY.y, mul2(vz, NZ.x))), mul2(rinv, rinv));  // cos_inc / r
    if (ATT) amp = mul2(amp, ex2_2(mul2(r, g.natt)));
    pr = mul2(amp, cs);
    pi = mul2(amp, sn);
}

// Centroid-relative forms of the two entries.  The point is given as
// D = p - c and R = |D| (c: the item's reference point, D rounded from the
// FP64 difference), the fragment as o = f - c and |o|^2 (formed once per
// chunk when its data is staged); r = |D - o| for the amplitude and the
// cosine.  The phase is k r = k R + k (r - R): the entry carries
// e^{ik (r - R)} with r - R = (|o|^2 - 2 o.D) / (r + R), free of
// cancellation, and e^{ik R} -- common to the point's row -- is applied in
// FP64 by the reduction (the host computes it from the FP64 R).  The
// readout's 1/r^2 term carries no phase, so the entry holds it times
// e^{-ik R} (the row's factor E, FP32).
// num = |o|^2 - 2 o.D = r^2 - R^2 (no cancellation); r^2 = R^2 + num is good
// to FP32's relative accuracy, enough for the amplitude, the cosine and r + R.
// The row's constants: D, R, R^2, E times 4 pi / k.
struct RelRow {
    f2 x, y, z, R, R2, Er, nEi;
};
__device__ __forceinline__ void rel_wave2(const Gen2 &g, const RelRow &p, f2 ox, f2 oy, f2 oz, f2 oo, f2 &r, f2 &rinv,
                                          f2 &sn, f2 &cs)
{
    const f2 num = fma2(dup2(-2.0f), fma2(ox, p.x, fma2(oy, p.y, mul2(oz, p.z))), oo);
    const f2 r2 = add2(p.R2, num);
    rinv = rsqrt2(r2);
    r = mul2(r2, rinv);
    const f2 s = add2(r, p.R);
    // the quotient from the approximate reciprocal, corrected by one Newton step
    const f2 y = rcp2(s);
    f2 dr = mul2(num, y);
    dr = fma2(y, fma2(dr ^ 0x8000000080000000ull, s, num), dr);
    const f2 f = fma2(dr, g.ph.khi, sub2(g.ph.magic, fma2(dr, g.ph.khi, g.ph.magic)));
    turns_sincos2(g.ph, fma2(dr, g.ph.klo, f), sn, cs);
}

template <bool ATT>
__device__ __forceinline__ void readout_rel2(const Gen2 &g, const float4 *F, const RelRow &p, f2 &gr, f2 &ngi)
{
    const ulonglong2 XY = ld2(F), ZA = ld2(F + 1), NXY = ld2(F + 4), NZ = ld2(F + 5);
    f2 r, rinv, sn, cs;
    rel_wave2(g, p, XY.x, XY.y, ZA.x, NZ.y, r, rinv, sn, cs);
    // cos_scat: (p - f).n / r
    const f2 d = fma2(sub2(p.x, XY.x), NXY.x, fma2(sub2(p.y, XY.y), NXY.y, mul2(sub2(p.z, ZA.x), NZ.x)));
    const f2 w = mul2(mul2(mul2(rinv, rinv), d), ZA.y);
    if (ATT) {
        const f2 e = ex2_2(mul2(r, g.natt));
        gr = mul2(w, fma2(e, fma2(g.qatt, cs, sn), mul2(rinv, p.Er)));
        ngi = mul2(w, fma2(e, fma2(g.nqatt, sn, cs), mul2(rinv, p.nEi)));
    } else {
        gr = mul2(w, fma2(rinv, p.Er, sn));
        ngi = mul2(w, fma2(rinv, p.nEi, cs));
    }
}

template <bool ATT>
__device__ __forceinline__ void incident_rel2(const Gen2 &g, const float4 *F, const RelRow &p, f2 &pr, f2 &pi)
{
    const ulonglong2 XY = ld2(F + 2), ZW = ld2(F + 3), NXY = ld2(F + 4), NZ = ld2(F + 5);
    f2 r, rinv, sn, cs;
    rel_wave2(g, p, XY.x, XY.y, ZW.x, ZW.y, r, rinv, sn, cs);
    // cos_inc / r: (q - s).n / r^2
    const f2 d = fma2(sub2(p.x, XY.x), NXY.x, fma2(sub2(p.y, XY.y), NXY.y, mul2(sub2(p.z, ZW.x), NZ.x)));
    f2 amp = mul2(d, mul2(rinv, rinv));
    if (ATT) amp = mul2(amp, ex2_2(mul2(r, g.natt)));
    pr = mul2(amp, cs);
    pi = mul2(amp, sn);
}

// The points of one thread for the current item: positions, or (relative
// phase) the row's constants.
struct RowPoints {
    f2 rx, ry, rz, qx, qy, qz;
    RelRow rel_rx, rel_src;
};

// four pairs of FP32 values -> (hi, lo) BF16 packed for a 16-byte row store
__device__ __forceinline__ uint32_t bf16x2(f2 v)
{
    float a, b;
    up2(v, a, b);
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ void split8(const f2 *x, uint4 &hi, uint4 &lo)
{
    uint32_t h[4], l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        h[q] = bf16x2(x[q]);
        l[q] = bf16x2(sub2(x[q], pk2(__uint_as_float(h[q] << 16), __uint_as_float(h[q] & 0xffff0000u))));
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ void st16(uint8_t *p, uint4 v) { *reinterpret_cast<uint4 *>(p) = v; }

// Operand stage of KC fragments: A (128 rows x 2KC) hi and lo, B (64 rows x
// 2KC) hi and lo, each row-group/k-group core matrix 128 bytes; element
// (row, k) of A at (k / 8) * 2048 + row * 16 + (k % 8) * 2.
template <int KC>
struct Stage {
    static constexpr int kA = 128 * 2 * KC * 2;  // bytes of one A copy (hi or lo)
    static constexpr int kB = 64 * 2 * KC * 2;
    static constexpr int kBytes = 2 * kA + 2 * kB;
    static constexpr int kLboA = 128 * 16, kLboB = 64 * 16;
};

// Fragment data of one chunk in shared memory, by pairs of fragments: readout
// centroids (x0 x1 y0 y1)(z0 z1 A0 A1), areas times k / (4 pi); source-hop
// centroids (x0 x1 y0 y1)(z0 z1 w0 w1); facet normals (x0 x1 y0 y1)(z0 z1 w0
// w1); and per fragment the visibility words (receiver bits x, y; source bits
// z, w).  Relative phase: centroids as offsets, |o|^2 of the source-hop
// centroid in its w, of the readout centroid in the normal's.
template <int KC>
struct ChunkFrags {
    float4 v[KC / 2][6];
    uint4 vis[KC];
};

// Element e (fragment e / 4, field e % 4) of chunk `chunk` of item it, zero
// past the item's fragments (their visibility words are zero, so padded
// fragments contribute nothing).  The relative phase stages it through
// stage_rel once the load has arrived.
__device__ __forceinline__ float4 fetch_frag(const BatchArgs &a, const BatchItem &it, int chunk, int kc, int e)
{
    const int n = chunk * kc + (e >> 2);
    if (n >= it.nfrag) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const long long g = (long long)it.frag0 + n;
    const int c = e & 3;
    const float4 *p = c == 0 ? a.frag_pos : c == 1 ? a.frag_spos : c == 2 ? a.frag_n
                                                                       : reinterpret_cast<const float4 *>(a.vis);
    // volatile: issued here, a chunk's generation ahead of its use (the
    // compiler otherwise moves the load down to it and every chunk waits for
    // memory)
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p + g));
    return v;
}

template <int KC, bool REL>
__device__ __forceinline__ void stage(ChunkFrags<KC> &F, const BatchItem &it, int e, float4 v)
{
    const int n = e >> 2, c = e & 3, h = n & 1;
    if (c == 3) {
        F.vis[n] = make_uint4(__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w));
        return;
    }
    float *d = reinterpret_cast<float *>(&F.v[n >> 1][2 * c]) + h;
    if (REL && c < 2) {
        v.x -= it.cx;
        v.y -= it.cy;
        v.z -= it.cz;
        const float oo = fmaf(v.x, v.x, fmaf(v.y, v.y, v.z * v.z));
        if (c == 1) v.w = oo;
        else *(reinterpret_cast<float *>(&F.v[n >> 1][5]) + 2 + h) = oo;  // the normal's thread leaves it alone
    }
    if (c == 0) v.w *= it.kr4pi;
    d[0] = v.x;
    d[2] = v.y;
    d[4] = v.z;
    if (!(REL && c == 2)) d[6] = v.w;
}

template <int KC, bool ATT, bool REL>
__device__ __forceinline__ void generate(uint8_t *st, const ChunkFrags<KC> &F, const Gen2 &g, int tid,
                                         const RowPoints &pt, bool rx_ok, bool src_ok)
{
    using S = Stage<KC>;
    uint8_t *Ahi = st, *Alo = st + S::kA, *Bhi = st + 2 * S::kA, *Blo = st + 2 * S::kA + S::kB;
    const int row = tid & 63;  // receiver (A) or source (B)
#pragma unroll 1
    for (int q = tid >> 6; q < KC / 8; q += kBatchThreads / 64) {
        f2 gr[4], ngi[4], pr[4], pi[4];
        // groups of kGenGroup fragment pairs: a group's entries are evaluated
        // without branches (independent chains the scheduler interleaves)
        // when any lane of the warp needs one of them, and selected by the
        // lane's bits; a group no lane needs is skipped
#pragma unroll
        for (int j0 = 0; j0 < 4; j0 += kGenGroup) {
            unsigned mrx = 0u, msrc = 0u;
#pragma unroll
            for (int j = 2 * j0; j < 2 * (j0 + kGenGroup); ++j) {
                const uint4 w4 = F.vis[8 * q + j];
                mrx |= (((row < 32 ? w4.x : w4.y) >> (row & 31)) & 1u) << (j - 2 * j0);
                msrc |= (((row < 32 ? w4.z : w4.w) >> (row & 31)) & 1u) << (j - 2 * j0);
            }
            if (!rx_ok) mrx = 0u;
            if (!src_ok) msrc = 0u;
#pragma unroll
            for (int j = j0; j < j0 + kGenGroup; ++j) gr[j] = ngi[j] = pr[j] = pi[j] = 0ull;
            if (__any_sync(0xffffffffu, mrx != 0u)) {
#pragma unroll
                for (int j = j0; j < j0 + kGenGroup; ++j) {
                    const float4 *f = F.v[4 * q + j];
                    f2 x, y;
                    if (REL) readout_rel2<ATT>(g, f, pt.rel_rx, x, y);
                    else readout2<ATT>(g, f, pt.rx, pt.ry, pt.rz, x, y);
                    gr[j] = pick2(x, mrx >> (2 * (j - j0)));
                    ngi[j] = pick2(y, mrx >> (2 * (j - j0)));
                }
            }
            if (__any_sync(0xffffffffu, msrc != 0u)) {
#pragma unroll
                for (int j = j0; j < j0 + kGenGroup; ++j) {
                    const float4 *f = F.v[4 * q + j];
                    f2 x, y;
                    if (REL) incident_rel2<ATT>(g, f, pt.rel_src, x, y);
                    else incident2<ATT>(g, f, pt.qx, pt.qy, pt.qz, x, y);
                    pr[j] = pick2(x, msrc >> (2 * (j - j0)));
                    pi[j] = pick2(y, msrc >> (2 * (j - j0)));
                }
            }
        }
        uint4 h, l;
        const int kr0 = q, ki0 = KC / 8 + q;  // k-groups of the real and imaginary halves
        // A row p:      [ Gr | -Gi ];  A row 64 + p: [ Gi | Gr ]
        split8(gr, h, l);
        st16(Ahi + kr0 * S::kLboA + row * 16, h);
        st16(Alo + kr0 * S::kLboA + row * 16, l);
        st16(Ahi + ki0 * S::kLboA + (64 + row) * 16, h);
        st16(Alo + ki0 * S::kLboA + (64 + row) * 16, l);
        split8(ngi, h, l);
        st16(Ahi + ki0 * S::kLboA + row * 16, h);
        st16(Alo + ki0 * S::kLboA + row * 16, l);
        // Gi: the same split with every sign bit flipped (exact)
        const uint4 sg = make_uint4(0x80008000u, 0x80008000u, 0x80008000u, 0x80008000u);
        st16(Ahi + kr0 * S::kLboA + (64 + row) * 16, make_uint4(h.x ^ sg.x, h.y ^ sg.y, h.z ^ sg.z, h.w ^ sg.w));
        st16(Alo + kr0 * S::kLboA + (64 + row) * 16, make_uint4(l.x ^ sg.x, l.y ^ sg.y, l.z ^ sg.z, l.w ^ sg.w));
        // B row q_src: [ Pr | Pi ]
        split8(pr, h, l);
        st16(Bhi + kr0 * S::kLboB + row * 16, h);
        st16(Blo + kr0 * S::kLboB + row * 16, l);
        split8(pi, h, l);
        st16(Bhi + ki0 * S::kLboB + row * 16, h);
        st16(Blo + ki0 * S::kLboB + row * 16, l);
    }
}

template <int KC, bool ATT, bool REL>
__global__ void __launch_bounds__(kBatchThreads, KC == 64 ? 1 : 2) k_batch(BatchArgs a)
{
    using S = Stage<KC>;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t tmem_base;
    __shared__ ChunkFrags<KC> sfrag[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tmem_alloc(&tmem_base, kTmemCols);
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int row = tid & 63;
    const bool rx_ok = row < a.nrx, src_ok = row < a.nsrc;
    const float4 rx4 = rx_ok ? a.rx[row] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float4 sq4 = src_ok ? a.src[row] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    RowPoints pt{};
    if (!REL) {
        pt.rx = dup2(rx4.x); pt.ry = dup2(rx4.y); pt.rz = dup2(rx4.z);
        pt.qx = dup2(sq4.x); pt.qy = dup2(sq4.y); pt.qz = dup2(sq4.z);
    }
    // the item's constants and the relative phase's point data of this thread's row
    Gen2 gen{};
    auto load_item = [&](int item, const BatchItem &it) {
        gen = gen2(it);
        if (!REL) return;
        const size_t q = (size_t)item * kBatchMaxPoints + row;
        const float4 D = __ldg(a.rel_rx + q), Q = __ldg(a.rel_src + q);
        const float2 E = __ldg(a.rel_rx_e + q);
        const float c = 1.0f / it.kr4pi;
        pt.rel_rx = RelRow{dup2(D.x), dup2(D.y), dup2(D.z), dup2(D.w), dup2(D.w * D.w), dup2(E.x * c), dup2(-E.y * c)};
        pt.rel_src = RelRow{dup2(Q.x), dup2(Q.y), dup2(Q.z), dup2(Q.w), dup2(Q.w * Q.w), 0ull, 0ull};
    };
    const uint32_t sbase = smem_u32(smem);
    const bool loader = tid < 4 * KC;  // thread tid stages element tid of each chunk's fragment data
    // this CTA's chunks: segments [g0, g1), chunk cc of segment sg
    const int g0 = a.cta_seg[blockIdx.x], g1 = a.cta_seg[blockIdx.x + 1];
    int sg = g0, cc = 0;
    int4 seg = make_int4(0, 0, 0, 0);
    BatchItem it{};
    if (sg < g1) {
        seg = a.segs[sg];
        it = a.items[seg.x];
        load_item(seg.x, it);
        if (loader) stage<KC, REL>(sfrag[0], it, tid, fetch_frag(a, it, seg.y, KC, tid));
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    uint32_t commits0 = 0, commits1 = 0;  // commits issued on each stage's barrier
    int last_st = -1;                     // stage of the most recent commit
    int local = 0;                        // chunks this CTA has generated
    bool ok = true;
    while (sg < g1 && ok) {
        const int st = local & 1;
        // the next chunk: its fragment data is loaded now and staged after this chunk's generation
        int nsg = sg, ncc = cc + 1;
        int4 nseg = seg;
        BatchItem nit = it;
        if (ncc >= seg.z) {
            nsg = sg + 1;
            ncc = 0;
            if (nsg < g1) {
                nseg = a.segs[nsg];
                nit = a.items[nseg.x];
            }
        }
        float4 nf = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (loader && nsg < g1) nf = fetch_frag(a, nit, nseg.y + ncc, KC, tid);
        // The operand stage is free once the MMAs that read it (two chunks back)
        // completed: each thread waits for itself, and a wait that ran out is
        // agreed on at the chunk's one barrier, before anything is issued.  (The
        // stage's next commit comes after that barrier, so no thread can miss a
        // phase; the fragment data written below were last read before the
        // previous one.)  With a barrier after the wait too, 16 scenes x 64 x 64 x
        // 8 frequencies took 1.17 ms against 1.085.
        bool done = true;
        if (local >= 2) {
            const uint32_t c = st ? commits1 : commits0;
            done = mbar_wait(&bar[st], (c - 1) & 1u);
        }
        generate<KC, ATT, REL>(smem + st * S::kBytes, sfrag[st], gen, tid, pt, rx_ok, src_ok);
        if (loader) stage<KC, REL>(sfrag[st ^ 1], nit, tid, nf);
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(done);
        if (!ok) break;
        if (tid == 0) {
            tc_fence_after();
            const uint32_t sA = sbase + st * S::kBytes, sB = sA + 2 * S::kA;
#pragma unroll
            for (int ks = 0; ks < 2 * KC / 16; ++ks) {
                const uint64_t ahi = sdesc(sA + ks * 2 * S::kLboA, S::kLboA, 128);
                const uint64_t alo = sdesc(sA + S::kA + ks * 2 * S::kLboA, S::kLboA, 128);
                const uint64_t bhi = sdesc(sB + ks * 2 * S::kLboB, S::kLboB, 128);
                const uint64_t blo = sdesc(sB + S::kB + ks * 2 * S::kLboB, S::kLboB, 128);
                mma_bf16(tmem, ahi, bhi, kIdesc, (cc > 0 || ks > 0) ? 1u : 0u);
                mma_bf16(tmem, ahi, blo, kIdesc, 1u);
                mma_bf16(tmem, alo, bhi, kIdesc, 1u);
            }
            mma_commit(&bar[st]);
        }
        if (st) ++commits1;
        else ++commits0;
        last_st = st;
        ++local;
        if (cc + 1 == seg.z) {
            // ---- segment end: the accumulator -> FP32 partial [128][64]
            const uint32_t c = st ? commits1 : commits0;
            const bool done = mbar_wait(&bar[st], (c - 1) & 1u);
            ok = __syncthreads_and(done);
            if (!ok) break;
            tc_fence_after();
            const int quarter = warp & 3, half = warp >> 2;
            const int drow = quarter * 32 + lane;
            float v[32];
            const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 32);
            tmem_ld16(taddr, v);
            tmem_ld16(taddr + 16, v + 16);
            float4 *out = reinterpret_cast<float4 *>(a.partial + ((long long)sg * 128 + drow) * 64 + half * 32);
#pragma unroll
            for (int q = 0; q < 8; ++q) out[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            tc_fence_before();
            __syncthreads();
        }
        if (nsg != sg && nsg < g1 && nseg.x != seg.x) load_item(nseg.x, nit);
        sg = nsg;
        cc = ncc;
        seg = nseg;
        it = nit;
    }
    // After a timed-out wait, MMAs committed earlier may still be writing the
    // accumulator and reading the operand stages.  tcgen05 operations of one
    // thread complete in issue order, so once the most recent commit has
    // arrived nothing is in flight: wait for it (bounded again) before the
    // tensor memory is released.  If that wait runs out as well, the tensor
    // memory is left allocated rather than released under a running MMA, and
    // the status says so (2).
    bool drained = true;
    if (!ok && last_st >= 0) {
        const uint32_t c = last_st ? commits1 : commits0;
        drained = __syncthreads_and(mbar_wait(&bar[last_st], (c - 1) & 1u));
    }
    if (!ok && tid == 0) atomicExch(a.status, drained ? 1 : 2);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0 && drained) tmem_dealloc(tmem, kTmemCols);
}

// Error-free sum of two FP32 values (Knuth's two-sum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e)
{
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// out[item][p][q] = sum over the item's segments in a fixed order, times
// the relative phase's row factors e^{ik R} of receiver p and source q when
// given.  The FP32 partials are added by compensated summation (a head and
// the sum of the two-sum error terms, all FP32: FP64 arithmetic is scarce on
// this part), the two words combined in FP64: the sum is exact to about
// 2^-46 of its terms' magnitude, as an FP64 accumulation would be for this
// many terms.  Grid (items, entry chunks): kRedShares threads per (receiver,
// source) entry, each with a contiguous share of the segments, the shares
// added in order (a thread that reads all of them one after the other is bound
// by that chain: 9 items of 34 segments 18 us, 11 in shares; 128 items of
// 17 take 36 us either way).
constexpr int kRedShares = 4;
__global__ void __launch_bounds__(256) k_batch_reduce(const float *partial, const int *item_seg_off,
                                                      const int *item_segs, int nrx, int nsrc, const double2 *erx,
                                                      const double2 *esrc, double2 *out)
{
    constexpr int kEnt = 256 / kRedShares;
    __shared__ float4 sS[kRedShares][kEnt];
    const int item = blockIdx.x, l = threadIdx.x % kEnt, g = threadIdx.x / kEnt;
    const int e = blockIdx.y * kEnt + l;
    const bool live = e < nrx * nsrc;
    const int s0 = item_seg_off[item], ns = item_seg_off[item + 1] - s0;
    const int p = live ? e / nsrc : 0, q = live ? e - p * nsrc : 0;
    float rh = 0.0f, rl = 0.0f, ih = 0.0f, il = 0.0f;
#pragma unroll 4
    for (int s = s0 + ns * g / kRedShares; s < s0 + ns * (g + 1) / kRedShares; ++s) {
        const float *P = partial + (long long)item_segs[s] * 128 * 64;
        float err;
        two_sum(rh, __ldg(P + p * 64 + q), rh, err);
        rl += err;
        two_sum(ih, __ldg(P + (64 + p) * 64 + q), ih, err);
        il += err;
    }
    sS[g][l] = make_float4(rh, rl, ih, il);
    __syncthreads();
    if (g > 0 || !live) return;
#pragma unroll
    for (int k = 1; k < kRedShares; ++k) {
        const float4 v = sS[k][l];
        float err;
        two_sum(rh, v.x, rh, err);
        rl += err + v.y;
        two_sum(ih, v.z, ih, err);
        il += err + v.w;
    }
    double re = (double)rh + (double)rl, im = (double)ih + (double)il;
    if (erx) {
        const double2 a = erx[item * kBatchMaxPoints + p], b = esrc[item * kBatchMaxPoints + q];
        const double er = a.x * b.x - a.y * b.y, ei = a.x * b.y + a.y * b.x;
        const double t = re * er - im * ei;
        im = re * ei + im * er;
        re = t;
    }
    out[(long long)item * nrx * nsrc + e] = make_double2(re, im);
}

}  // namespace

size_t batch_smem_bytes(int kc)
{
    return kc == 64 ? (size_t)2 * Stage<64>::kBytes
                    : kc == 32 ? (size_t)2 * Stage<32>::kBytes : (size_t)2 * Stage<16>::kBytes;
}

namespace {
template <int KC>
cudaError_t prepare_k()
{
    const int sm = (int)batch_smem_bytes(KC);
    cudaError_t e = cudaFuncSetAttribute(k_batch<KC, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_batch<KC, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_batch<KC, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_batch<KC, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
    return e;
}
}  // namespace

cudaError_t batch_prepare()
{
    cudaError_t e = prepare_k<32>();
    if (e == cudaSuccess) e = prepare_k<64>();
    if (e == cudaSuccess) e = prepare_k<16>();
    return e;
}

namespace {
template <int KC>
void launch_k(const BatchArgs &a, int grid, size_t sm, bool att, bool rel, cudaStream_t s)
{
    if (att) {
        if (rel) k_batch<KC, true, true><<<grid, kBatchThreads, sm, s>>>(a);
        else k_batch<KC, true, false><<<grid, kBatchThreads, sm, s>>>(a);
    } else {
        if (rel) k_batch<KC, false, true><<<grid, kBatchThreads, sm, s>>>(a);
        else k_batch<KC, false, false><<<grid, kBatchThreads, sm, s>>>(a);
    }
}
}  // namespace

void launch_batch(const BatchArgs &a, int kc, int grid, bool att, cudaStream_t s)
{
    const size_t sm = batch_smem_bytes(kc);
    if (grid <= 0) return;
    const bool rel = a.rel_rx != nullptr;
    if (kc == 64) launch_k<64>(a, grid, sm, att, rel, s);
    else if (kc == 16) launch_k<16>(a, grid, sm, att, rel, s);
    else launch_k<32>(a, grid, sm, att, rel, s);
}

void launch_batch_reduce(const float *partial, const int *item_seg_off, const int *item_segs, int nitems, int nrx,
                         int nsrc, const double2 *erx, const double2 *esrc, double2 *out, cudaStream_t s)
{
    if (nitems > 0)
        k_batch_reduce<<<dim3(nitems, (nrx * nsrc * kRedShares + 255) / 256), 256, 0, s>>>(
            partial, item_seg_off, item_segs, nrx, nsrc, erx, esrc, out);
}

}  // namespace sonar
