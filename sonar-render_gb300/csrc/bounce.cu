// bounce.cu -- the symmetric bounce sum (FACET_SELF with reciprocity).
//
// Evaluated once per unordered pair, as the reference does (OptiX.cu:367-390):
// for source tile I < destination tile J the CTA computes T_ij = 0.9-free
// G(r_ij) cos_scat cos_inc once per pair and adds T_ij w_i into its
// destination row j (registers) and T_ij w_j into the column of i (a
// shared-memory transpose per warp, per-warp shared sums, one write per
// (I, J)).  Tiles are in facet order, so every interacting pair of such a
// block has facet(i) < facet(j): the row term is the forward term and the
// column term the reciprocal one, dropped in the final reduction when
// P_in[i] == 0.  The diagonal tile (I == J) runs the destination-owned loop.
// Column sums of (I, J) land at colpart[256 J (J-1) / 2 + i];
// k_finalize_f2f_sym adds them in a fixed order (deterministic results).
//
// Blocks come in two kinds.  PLANAR blocks: every pair interacts (class ALL),
// each tile lies on one facet, no pair can be closer than r_min.  There
// r cos_scat is the distance of p_j from the source tile's plane and
// r cos_inc that of p_i from the destination tile's plane, so both factors
// leave the pair loop: T_ij = d1(j) d2(i) g(r_ij).  What is left per pair --
// the distance, its phase, g and the two complex multiply-adds -- is packed
// two sources to a register (pack2.cuh), two destinations to a thread, so
// that the source data's shared loads and the column transpose are paid once
// per two destinations.  GENERAL blocks (per-pair bits, gates to evaluate,
// tiles of several facets) take both cosines from the pair's own vector, in
// the same packed form, one destination to a thread.  The diagonal and the
// blocks that reach r_min run the scalar arithmetic of sym_pair.
//
// What bounds it: FP32 lanes, about 29 operations of a planar pair (38 of a
// general one) against 32 lanes per clock and scheduler, beside 3
// special-function operations at 4 lanes; the scalar form of every block was
// bound by issue, about 57 instructions a pair.  FACET_SELF of the 60 kHz
// trihedral (6.4e9 unordered pairs, 152 SMs): 11.97 ms
// scalar, 6.80 ms in this form (40 kHz: 2.53 -> 1.60, 30 kHz: 0.91 -> 0.56).
// Measured and left out: sums over the blocks and warps in two FP32 words (6.74
// ms, but fewer bits than FP64 and NaN for infinite terms), and with them three
// CTAs per SM (7.05 ms), five (7.3 ms), the pair loop unrolled by 1 or 4 (the
// same time); integer conversions to FP64 (6.83).
#include "sonar_internal.h"
#include "green.cuh"
#include "pack2.cuh"

#include <algorithm>
#include <climits>

namespace sonar {
namespace {

constexpr int kSymThreads = 128;
constexpr int kSymWarps = kSymThreads / 32;
// Shared-memory transpose of one warp's column terms, 16 sources at a time.
// Other blocks: row = lane (destination), column = source, pitch 17 float2;
// planar blocks: column = source pair, pitch 9 float4.  Both keep the
// row-wise writes and the column-wise reads free of bank conflicts.
constexpr int kTrPitch = 17, kTrPitch4 = 9;
constexpr size_t kSymTrBytes = sizeof(float4) * kSymWarps * 32 * kTrPitch4;
static_assert(kSymTrBytes >= sizeof(float2) * kSymWarps * 32 * kTrPitch, "both transposes fit");
constexpr size_t kSymDynSmem = kSymTrBytes + sizeof(float2) * 2 * kSymWarps * kTile;

// ---------------------------------------------------------------- scalar blocks
// one 32-source word of an off-diagonal block: row terms into the thread's
// destination, column terms summed over the warp into colw[word].
template <bool ATT, bool GATE>
__device__ __forceinline__ void sym_word(const SumArgs &a, const float4 *sA, const float4 *sB, int w, uint32_t m,
                                         const Dst &d, float wjr, float wji, float &fr, float &fi, float2 *colw,
                                         float2 *tr, int lane)
{
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll 4
        for (int b = 0; b < 16; ++b) {
            const int q = w * 32 + h * 16 + b;
            const float4 A = sA[q], B = sB[q];
            float Tr, Ti;
            bool ok;
            sym_pair<ATT, GATE, true>(a, A, B, d, Tr, Ti, ok);
            const bool on = ((m >> (h * 16 + b)) & 1u) && ok;
            Tr = on ? Tr : 0.0f;
            Ti = on ? Ti : 0.0f;
            fr = fmaf(Tr, A.w, fmaf(-Ti, B.w, fr));  // forward term into this destination
            fi = fmaf(Tr, B.w, fmaf(Ti, A.w, fi));
            tr[lane * kTrPitch + b] = make_float2(Tr * wjr - Ti * wji, Tr * wji + Ti * wjr);  // reciprocal term
        }
        __syncwarp();
        // lane l sums column (l & 15) over rows 16 (l >> 4) .. +15; the two halves combine
        const int c = lane & 15, r0 = (lane >> 4) * 16;
        float sr = 0.0f, si = 0.0f;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float2 v = tr[(r0 + r) * kTrPitch + c];
            sr += v.x;
            si += v.y;
        }
        sr += __shfl_xor_sync(0xffffffffu, sr, 16);
        si += __shfl_xor_sync(0xffffffffu, si, 16);
        if (lane < 16) colw[w * 32 + h * 16 + lane] = make_float2(sr, si);
        __syncwarp();
    }
}

template <bool ATT, bool GATE>
__device__ __forceinline__ void diag_word(const SumArgs &a, const float4 *sA, const float4 *sB, int w, uint32_t m,
                                          const Dst &d, float &fr, float &fi)
{
#pragma unroll 4
    for (int b = 0; b < 32; ++b) {
        const float4 A = sA[w * 32 + b], B = sB[w * 32 + b];
        float Tr, Ti;
        bool ok;
        sym_pair<ATT, GATE, true>(a, A, B, d, Tr, Ti, ok);
        const bool on = ((m >> b) & 1u) && ok;
        Tr = on ? Tr : 0.0f;
        Ti = on ? Ti : 0.0f;
        fr = fmaf(Tr, A.w, fmaf(-Ti, B.w, fr));
        fi = fmaf(Tr, B.w, fmaf(Ti, A.w, fi));
    }
}

// ---------------------------------------------------------------- packed blocks
// Column sums of 16 sources: tr[destination lane][source pair] holds (Re0
// Re1 Im0 Im1); lane l sums source pair (l & 7) over rows 8 (l >> 3) .. +7,
// the four groups combine, col gets the 16 sums of the warp.
__device__ __forceinline__ void reduce_pairs(const float4 *tr, float2 *col, int lane)
{
    __syncwarp();
    const int c = lane & 7, r0 = (lane >> 3) * 8;
    ulonglong2 s = *reinterpret_cast<const ulonglong2 *>(&tr[r0 * kTrPitch4 + c]);
#pragma unroll
    for (int r = 1; r < 8; ++r) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(&tr[(r0 + r) * kTrPitch4 + c]);
        s.x = add2(s.x, v.x);
        s.y = add2(s.y, v.y);
    }
#pragma unroll
    for (int o = 8; o <= 16; o <<= 1) {
        s.x = add2(s.x, __shfl_xor_sync(0xffffffffu, s.x, o));
        s.y = add2(s.y, __shfl_xor_sync(0xffffffffu, s.y, o));
    }
    if (lane < 8) {
        float re0, re1, im0, im1;
        up2(s.x, re0, re1);
        up2(s.y, im0, im1);
        *reinterpret_cast<float4 *>(&col[2 * c]) = make_float4(re0, im0, re1, im1);
    }
    __syncwarp();
}

// g(r) = Tr - i Ti of two pairs, times f: (1 / r^3) [sin kr + (4 pi / k) / r
// - i cos kr], the constant k / (4 pi) left to the caller; with attenuation
// the sine and cosine carry e^{-ka r} and the terms of ka / k.
struct Green2 {
    Phase2 ph;
    f2 c4pik, natt, qatt, nqatt;
};
__device__ __forceinline__ Green2 green2(const SumArgs &a)
{
    return Green2{phase2(a.k2hi, a.k2lo), dup2(1.0f / a.kr4pi), dup2(-a.ka * 1.44269504088896341f),
                  dup2(a.ka / a.kr), dup2(-(a.ka / a.kr))};
}
template <bool ATT, bool FACTOR>
__device__ __forceinline__ void green_pair2(const Green2 &g, f2 r2, f2 rinv, f2 f, f2 &Tr, f2 &Ti)
{
    const f2 r0 = mul2(r2, rinv);
    f2 sn, cs;
    sincos2(g.ph, r0, rinv, sn, cs);
    const f2 rinv2 = mul2(rinv, rinv);
    f2 osc = mul2(rinv2, rinv);
    if (FACTOR) osc = mul2(osc, f);
    if (ATT) {
        f2 st = mul2(osc, mul2(rinv, g.c4pik));
        osc = mul2(osc, ex2_2(mul2(r0, g.natt)));
        Tr = fma2(osc, fma2(g.qatt, cs, sn), st);
        Ti = mul2(osc, fma2(g.nqatt, sn, cs));
    } else {
        Tr = mul2(osc, fma2(rinv, g.c4pik, sn));
        Ti = mul2(osc, cs);
    }
}

// Planar blocks: both destinations of the thread against the source words
// [w0, w1): sXY, sZW, sWi hold source pairs (x0 x1 y0 y1), (z0 z1 wr0 wr1),
// (wi0 wi1 ..), the row weights with d2(i) in them; wr, wi, nwr = -wr the
// destinations' column weights with d1(j).
// Rows: racc[d] = (Re, first and second part of Im); columns into colw.
struct PlanarDst {
    f2 x, y, z, wr, wi, nwr;
};

template <bool ATT>
__device__ __forceinline__ void planar_words(const Green2 &g, const float4 *sXY, const float4 *sZW, const float4 *sWi,
                                             int w0, int w1, const PlanarDst (&d)[2], f2 (&racc)[2][3], float2 *colw,
                                             float4 *tr, int lane)
{
    for (int h = 2 * w0; h < 2 * w1; ++h) {
#pragma unroll 2
        for (int b = 0; b < 8; ++b) {
            const ulonglong2 XY = *reinterpret_cast<const ulonglong2 *>(&sXY[h * 8 + b]);
            const ulonglong2 ZW = *reinterpret_cast<const ulonglong2 *>(&sZW[h * 8 + b]);
            const f2 WI = *reinterpret_cast<const f2 *>(&sWi[h * 8 + b]);
            f2 cr = 0ull, ci = 0ull;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const f2 vx = sub2(d[q].x, XY.x), vy = sub2(d[q].y, XY.y), vz = sub2(d[q].z, ZW.x);
                const f2 r2 = fma2(vx, vx, fma2(vy, vy, mul2(vz, vz)));
                f2 Tr, Ti;
                green_pair2<ATT, false>(g, r2, rsqrt2(r2), 0ull, Tr, Ti);
                // T w with T = Tr - i Ti
                racc[q][0] = fma2(Tr, ZW.y, fma2(Ti, WI, racc[q][0]));
                racc[q][1] = fma2(Tr, WI, racc[q][1]);
                racc[q][2] = fma2(Ti, ZW.y, racc[q][2]);
                if (q == 0) {
                    cr = fma2(Tr, d[q].wr, mul2(Ti, d[q].wi));
                    ci = fma2(Tr, d[q].wi, mul2(Ti, d[q].nwr));
                } else {
                    cr = fma2(Tr, d[q].wr, fma2(Ti, d[q].wi, cr));
                    ci = fma2(Tr, d[q].wi, fma2(Ti, d[q].nwr, ci));
                }
            }
            *reinterpret_cast<ulonglong2 *>(&tr[lane * kTrPitch4 + b]) = make_ulonglong2(cr, ci);
        }
        reduce_pairs(tr, colw + h * 16, lane);
    }
}

// General blocks: one destination of the thread against one 32-source word:
// sA holds the pairs (x0 x1 y0 y1) and, 128 entries on, (z0 z1 wr0 wr1); sB
// (nx0 nx1 ny0 ny1) and (nz0 nz1 wi0 wi1).  MODE 0: every pair interacts; 1:
// the pairs of m; 2: those of m whose cosine gates pass (the estimate decides
// outside its band, the exact expression inside it).  T's sign is flipped
// (the factor is d1 d2 = -(r cos_scat)(r cos_inc)): the caller's constant is
// -k / (4 pi).
template <bool ATT, int MODE>
__device__ __forceinline__ void general_word(const Green2 &g, const float4 *sA, const float4 *sB, int w, uint32_t m,
                                             const Dst &p, const PlanarDst &d, f2 nx, f2 ny, f2 nz, f2 (&racc)[3],
                                             float2 *colw, float4 *tr, int lane)
{
#pragma unroll 1
    for (int h = 2 * w; h < 2 * w + 2; ++h) {
#pragma unroll 2
        for (int b = 0; b < 8; ++b) {
            const int q = h * 8 + b;
            const ulonglong2 XY = *reinterpret_cast<const ulonglong2 *>(&sA[q]);
            const ulonglong2 ZW = *reinterpret_cast<const ulonglong2 *>(&sA[kSymThreads + q]);
            const ulonglong2 NN = *reinterpret_cast<const ulonglong2 *>(&sB[q]);
            const ulonglong2 NW = *reinterpret_cast<const ulonglong2 *>(&sB[kSymThreads + q]);
            const f2 vx = sub2(d.x, XY.x), vy = sub2(d.y, XY.y), vz = sub2(d.z, ZW.x);
            const f2 r2 = fma2(vx, vx, fma2(vy, vy, mul2(vz, vz)));
            const f2 rinv = rsqrt2(r2);
            const f2 d1 = fma2(vx, NN.x, fma2(vy, NN.y, mul2(vz, NW.x)));  // r cos_scat
            const f2 d2 = fma2(vx, nx, fma2(vy, ny, mul2(vz, nz)));        // -r cos_inc
            f2 Tr, Ti;
            green_pair2<ATT, true>(g, r2, rinv, mul2(d1, d2), Tr, Ti);
            if (MODE > 0) {
                bool on0 = (m >> (2 * b)) & 1u, on1 = (m >> (2 * b + 1)) & 1u;
                if (MODE == 2) {
                    float a0, a1, c0, c1;
                    up2(mul2(d1, rinv), a0, a1);
                    up2(mul2(d2, rinv), c0, c1);
                    const bool sure0 = fminf(a0, -c0) > 2e-6f || fminf(a0, -c0) < 0.0f;
                    const bool sure1 = fminf(a1, -c1) > 2e-6f || fminf(a1, -c1) < 0.0f;
                    bool p0 = fminf(a0, -c0) > 2e-6f, p1 = fminf(a1, -c1) > 2e-6f;
                    if (__any_sync(0xffffffffu, (on0 && !sure0) || (on1 && !sure1))) {
                        float x0, x1, y0, y1, z0, z1, u0, u1, v0, v1, w0, w1;
                        up2(vx, x0, x1);
                        up2(vy, y0, y1);
                        up2(vz, z0, z1);
                        up2(NN.x, u0, u1);
                        up2(NN.y, v0, v1);
                        up2(NW.x, w0, w1);
                        p0 = gate_est(a0, x0, y0, z0, 1.0f, u0, v0, w0) &&
                             gate_est(-c0, x0, y0, z0, -1.0f, p.nx, p.ny, p.nz);
                        p1 = gate_est(a1, x1, y1, z1, 1.0f, u1, v1, w1) &&
                             gate_est(-c1, x1, y1, z1, -1.0f, p.nx, p.ny, p.nz);
                    }
                    on0 = on0 && p0;
                    on1 = on1 && p1;
                }
                float r0, r1, i0, i1;
                up2(Tr, r0, r1);
                up2(Ti, i0, i1);
                Tr = pk2(on0 ? r0 : 0.0f, on1 ? r1 : 0.0f);
                Ti = pk2(on0 ? i0 : 0.0f, on1 ? i1 : 0.0f);
            }
            racc[0] = fma2(Tr, ZW.y, fma2(Ti, NW.y, racc[0]));
            racc[1] = fma2(Tr, NW.y, racc[1]);
            racc[2] = fma2(Ti, ZW.y, racc[2]);
            *reinterpret_cast<ulonglong2 *>(&tr[lane * kTrPitch4 + b]) =
                make_ulonglong2(fma2(Tr, d.wr, mul2(Ti, d.wi)), fma2(Tr, d.wi, mul2(Ti, d.nwr)));
        }
        m >>= 16;
        reduce_pairs(tr, colw + h * 16, lane);
    }
}

// ---------------------------------------------------------------- work list
// Can a block's pairs take the packed forms?  No pair near the
// regularisation radius (nor, by it, at a distance FP32 squares to a
// denormal), and magnitudes that FP32 holds.
__device__ __forceinline__ bool packable(const SumArgs &a, const TileGeom &I, const TileGeom &J)
{
    const float gap = box_gap(I.lo, I.hi, J.lo, J.hi);
    if (!(gap > fmaxf(a.rmin * 1.001f, 1e-9f))) return false;
    return fmaxf(box_extent(I.lo, I.hi), box_extent(J.lo, J.hi)) < 1e6f &&
           packed_in_range(a, gap, box_diag(I.lo, I.hi, J.lo, J.hi), fmaxf(I.wmax, J.wmax));
}

// The non-empty blocks of destination row J (source tiles t <= J whose flag
// is not NONE) in tile order: blist[J * ntiles + k] from the front the general
// and scalar blocks, from the back (k = 0 last) the planar ones; rowcnt their
// counts.
__global__ void __launch_bounds__(kTile) k_sym_rows(SumArgs a, int ntiles, int nb, int packed_ok, int *blist,
                                                   int2 *rowcnt)
{
    __shared__ int sWarp[2][kTile / 32];
    const int J = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tmax = min(J, ntiles - 1);
    const TileGeom gJ = a.geom[J];
    int *row = blist + (long long)J * ntiles;
    int base0 = 0, base1 = 0;
    for (int t0 = 0; t0 <= tmax; t0 += kTile) {
        const int t = t0 + tid;
        const uint8_t fl = t <= tmax ? a.mask.flags[(long long)t * nb + J] : kFlagNone;
        const bool on = fl != kFlagNone;
        bool pl = packed_ok && fl == kFlagAll && t < J && gJ.n.w != 0.0f;
        if (pl) {
            const TileGeom gI = a.geom[t];
            pl = gI.n.w != 0.0f && packable(a, gI, gJ);
        }
        const unsigned b0 = __ballot_sync(0xffffffffu, on && !pl), b1 = __ballot_sync(0xffffffffu, pl);
        if (lane == 0) {
            sWarp[0][warp] = __popc(b0);
            sWarp[1][warp] = __popc(b1);
        }
        __syncthreads();
        int off0 = 0, off1 = 0, tot0 = 0, tot1 = 0;
#pragma unroll
        for (int w = 0; w < kTile / 32; ++w) {
            off0 += w < warp ? sWarp[0][w] : 0;
            off1 += w < warp ? sWarp[1][w] : 0;
            tot0 += sWarp[0][w];
            tot1 += sWarp[1][w];
        }
        const unsigned below = (1u << lane) - 1u;
        if (on && !pl) row[base0 + off0 + __popc(b0 & below)] = t;
        if (pl) row[ntiles - 1 - (base1 + off1 + __popc(b1 & below))] = t;
        base0 += tot0;
        base1 += tot1;
        __syncthreads();
    }
    if (tid == 0) rowcnt[J] = make_int2(base0, base1);
}

// chunks of cnt blocks: per blocks to a chunk, or (sub > 1) sub chunks to a block
__device__ __forceinline__ int chunk_count(int cnt, int per, int sub) { return sub > 1 ? cnt * sub : (cnt + per - 1) / per; }

// Exclusive scans of the rows' chunk counts (general chunks off[J].x, planar
// ones off[J].y; off[nb] the totals); nchunks: all, general, the next-chunk
// counter of the sum, zeroed, and the blocks per chunk that were taken: the
// shape's, or two where those make more chunks than the partials have room
// for.  One CTA of 1024 threads.
__global__ void __launch_bounds__(1024) k_sym_scan(const int2 *rowcnt, int nb, SymShape sh, int cap, int2 *off,
                                                  int *nchunks)
{
    __shared__ int2 sW[32];
    __shared__ int2 sCarry;
    __shared__ int sTotal;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        sCarry = make_int2(0, 0);
        sTotal = 0;
    }
    __syncthreads();
    int mine = 0;
    for (int J = tid; J < nb; J += 1024) {
        const int2 cnt = rowcnt[J];
        mine += chunk_count(cnt.x, sh.per_general, sh.sub) + chunk_count(cnt.y, sh.per_planar, sh.sub);
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) atomicAdd(&sTotal, mine);
    __syncthreads();
    if (sTotal > cap) {
        sh.per_general = max(sh.per_general, 2);
        sh.per_planar = max(sh.per_planar, 2);
    }
    for (int J0 = 0; J0 < nb; J0 += 1024) {
        const int J = J0 + tid;
        const int2 cnt = J < nb ? rowcnt[J] : make_int2(0, 0);
        const int2 n = make_int2(chunk_count(cnt.x, sh.per_general, sh.sub), chunk_count(cnt.y, sh.per_planar, sh.sub));
        int2 v = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, v.x, o), y = __shfl_up_sync(0xffffffffu, v.y, o);
            if (lane >= o) {
                v.x += x;
                v.y += y;
            }
        }
        if (lane == 31) sW[warp] = v;
        __syncthreads();
        if (warp == 0) {
            int2 x = sW[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int p = __shfl_up_sync(0xffffffffu, x.x, o), q = __shfl_up_sync(0xffffffffu, x.y, o);
                if (lane >= o) {
                    x.x += p;
                    x.y += q;
                }
            }
            sW[lane] = x;
        }
        __syncthreads();
        const int2 pre = warp > 0 ? sW[warp - 1] : make_int2(0, 0);
        const int2 excl = make_int2(sCarry.x + pre.x + v.x - n.x, sCarry.y + pre.y + v.y - n.y);
        if (J < nb) off[J] = excl;
        __syncthreads();
        if (tid == 1023) sCarry = make_int2(excl.x + n.x, excl.y + n.y);
        __syncthreads();
    }
    if (tid == 0) {
        off[nb] = sCarry;
        nchunks[0] = sCarry.x + sCarry.y;
        nchunks[1] = sCarry.x;
        nchunks[2] = 0;
        nchunks[3] = sh.per_general;
        nchunks[4] = sh.per_planar;
    }
}

// The chunks of row J: general ones at off[J].x, planar ones at nchunks[1] +
// off[J].y (general chunks, the dearer ones, are taken first).  A chunk:
// (J, first block, end block | first word << 20 | end word << 24, planar).
__global__ void __launch_bounds__(128) k_sym_fill(const int2 *rowcnt, const int2 *off, const int *nchunks, int sub,
                                                 int4 *chunks)
{
    const int J = blockIdx.x;
    const int2 cnt = rowcnt[J], o = off[J];
    for (int kind = 0; kind < 2; ++kind) {
        const int c = kind ? cnt.y : cnt.x, per = nchunks[3 + kind];
        const int n = chunk_count(c, per, sub), base = kind ? nchunks[1] + o.y : o.x;
        const int words = kWordsPerTile / sub;
        for (int k = threadIdx.x; k < n; k += blockDim.x) {
            const int k0 = sub > 1 ? k / sub : k * per;
            const int k1 = sub > 1 ? k0 + 1 : min(c, k0 + per);
            const int w0 = sub > 1 ? (k % sub) * words : 0, w1 = w0 + words;
            chunks[base + k] = make_int4(J, k0, k1 | (w0 << 20) | (w1 << 24), kind);
        }
    }
}

// ---------------------------------------------------------------- the sum
// Persistent CTAs of 128 threads (destinations tid and tid + 128 of the row's
// tile) take the chunks from a counter in chunk order, so chunks of uneven
// cost balance over the CTAs; every chunk writes its own output locations, so
// the results do not depend on which CTA took it.  Per chunk: the row terms
// of its blocks into rowpart[chunk], the column terms of block (t, J), t < J,
// into colpart[256 J (J-1) / 2 + i].  Tile sums are FP32, what adds them up
// (over the blocks of a chunk, over the warps of a column) FP64.
// Four CTAs per SM: 128 registers a thread, which the planar loop's two
// destinations fill.
template <bool ATT>
__global__ void __launch_bounds__(kSymThreads, 4) k_sum_f2f_sym(SumArgs a, SymWork wl, double2 *colpart,
                                                                double2 *rowpart)
{
    extern __shared__ float4 sDyn[];  // kSymDynSmem bytes: per-warp transpose tiles, then column sums
    __shared__ float4 sA[kTile];      // packed: pairs (x0 x1 y0 y1) | (z0 z1 wr0 wr1)
    __shared__ float4 sB[kTile];      // planar: pairs (wi0 wi1 d2_0 d2_1); general: normals and wi
    __shared__ int sCh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float4 *const tr4 = sDyn + warp * 32 * kTrPitch4;
    float2 *const tr2 = reinterpret_cast<float2 *>(tr4);
    float2(*const sCol)[kTile] = reinterpret_cast<float2(*)[kTile]>(sDyn + kSymTrBytes / sizeof(float4));
    const int nch = *wl.nchunks;
    for (;;) {
        __syncthreads();  // the previous chunk is done with sCh and the shared arrays
        if (tid == 0) sCh = atomicAdd(wl.next, 1);
        __syncthreads();
        const int ch = sCh;
        if (ch >= nch) break;  // CTA-uniform
        const int4 cw = wl.chunks[ch];
        const int J = cw.x, k0 = cw.y, k1 = cw.z & 0xfffff, wA = (cw.z >> 20) & 15, wB = (cw.z >> 24) & 15;
        const long long cbase = (long long)kTile * J * (J - 1) / 2;  // this J's column region
        const int *row = wl.blist + (long long)J * wl.ntiles;
        double accr[2] = {0.0, 0.0}, acci[2] = {0.0, 0.0};
        if (cw.w) {
            // ---- planar blocks
            const Green2 g = green2(a);
            const TileGeom gJ = a.geom[J];
            float px[2], py[2], pz[2], wr[2], wi[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = J * kTile + q * kSymThreads + tid;
                const bool live = j < a.ndst;
                const float4 A = a.srcA[live ? j : J * kTile];
                px[q] = A.x; py[q] = A.y; pz[q] = A.z;
                wr[q] = live ? A.w : 0.0f;
                wi[q] = live ? a.srcB[j].w : 0.0f;
            }
            for (int kk = k0; kk < k1; ++kk) {
                const int t = row[wl.ntiles - 1 - kk];
                const TileGeom gI = a.geom[t];
                const int i0 = t * kTile;
                if (kk > k0) __syncthreads();
                {
                    // source pair tid: positions, row weights times d2(i); past the end the
                    // tile's first position with weight 0
                    float4 A[2];
                    float v[2], d2[2];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int i = i0 + 2 * tid + s;
                        const bool in = i < a.nsrc;
                        A[s] = a.srcA[in ? i : i0];
                        v[s] = in ? a.srcB[i].w : 0.0f;
                        if (!in) A[s].w = 0.0f;
                        // r cos_inc = -(p_j - p_i).n_j: p_i's distance from the destination plane
                        d2[s] = plane_distance(gJ, A[s].x, A[s].y, A[s].z);
                    }
                    sA[tid] = make_float4(A[0].x, A[1].x, A[0].y, A[1].y);
                    sA[kSymThreads + tid] = make_float4(A[0].z, A[1].z, A[0].w * d2[0], A[1].w * d2[1]);
                    sB[tid] = make_float4(v[0] * d2[0], v[1] * d2[1], d2[0], d2[1]);
                }
                PlanarDst d[2];
                float d1[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    d1[q] = plane_distance(gI, px[q], py[q], pz[q]);  // r cos_scat
                    d[q] = PlanarDst{dup2(px[q]), dup2(py[q]), dup2(pz[q]), dup2(wr[q] * d1[q]), dup2(wi[q] * d1[q]),
                                     dup2(-(wr[q] * d1[q]))};
                }
                f2 racc[2][3] = {{0ull, 0ull, 0ull}, {0ull, 0ull, 0ull}};
                __syncthreads();
                planar_words<ATT>(g, sA, sA + kSymThreads, sB, wA, wB, d, racc, &sCol[warp][0], tr4, lane);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float s1 = a.kr4pi * d1[q];
                    accr[q] += (double)(s1 * sum2(racc[q][0]));
                    acci[q] += (double)(s1 * (sum2(racc[q][1]) - sum2(racc[q][2])));
                }
                __syncthreads();
                // column sums over the four warps, times d2(i)
                const int i = 2 * tid;  // this thread's source pair
                if (i >= wA * 32 && i < wB * 32) {
                    const float4 D = sB[tid];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        double sr = (double)sCol[0][i + s].x, si = (double)sCol[0][i + s].y;
#pragma unroll
                        for (int k = 1; k < kSymWarps; ++k) {
                            const float2 v = sCol[k][i + s];
                            sr += (double)v.x;
                            si += (double)v.y;
                        }
                        const double f = (double)(a.kr4pi * (s ? D.w : D.z));
                        colpart[cbase + i0 + i + s] = make_double2(sr * f, si * f);
                    }
                }
            }
        } else {
            // ---- general and scalar blocks, one half of the row's destinations at a time
            const Green2 g = green2(a);
            const TileGeom gJ = a.geom[J];
            for (int kk = k0; kk < k1; ++kk) {
                const int t = row[kk];
                const TileGeom gI = a.geom[t];
                const uint8_t fl = a.mask.flags[(long long)t * a.mask.ndstblocks + J];
                const int i0 = t * kTile;
                const bool packed = wl.packed_ok && t < J && packable(a, gI, gJ);
                if (kk > k0) __syncthreads();
                if (packed) {
                    // source pair tid; past the end the tile's first fragment with weight 0
                    float4 A[2], B[2];
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const int i = i0 + 2 * tid + s;
                        const bool in = i < a.nsrc;
                        A[s] = a.srcA[in ? i : i0];
                        B[s] = a.srcB[in ? i : i0];
                        if (!in) A[s].w = B[s].w = 0.0f;
                    }
                    sA[tid] = make_float4(A[0].x, A[1].x, A[0].y, A[1].y);
                    sA[kSymThreads + tid] = make_float4(A[0].z, A[1].z, A[0].w, A[1].w);
                    sB[tid] = make_float4(B[0].x, B[1].x, B[0].y, B[1].y);
                    sB[kSymThreads + tid] = make_float4(B[0].z, B[1].z, B[0].w, B[1].w);
                } else {
                    for (int s = tid; s < kTile; s += kSymThreads) {
                        const int i = i0 + s;
                        const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        sA[s] = i < a.nsrc ? a.srcA[i] : z;
                        sB[s] = i < a.nsrc ? a.srcB[i] : z;
                    }
                }
                __syncthreads();
                const int ntile = min(kTile, a.nsrc - i0);
                const int nw = min((ntile + 31) >> 5, wB);
                const bool gate = fl == kFlagClear;
                const float flip = -a.kr4pi;
#pragma unroll 1
                for (int half = 0; half < 2; ++half) {
                    const int j = J * kTile + half * kSymThreads + tid;
                    const bool live = j < a.ndst;
                    int limit = a.nsrc;
                    // a dead thread takes the row's first destination with weight 0
                    float4 p = a.srcA[live ? j : J * kTile], n = a.srcB[live ? j : J * kTile];
                    if (live) limit = a.dst_limit[j];
                    else p.w = n.w = 0.0f;
                    const Dst d{p.x, p.y, p.z, n.x, n.y, n.z};
                    const float wjr = p.w, wji = n.w;  // this destination's own source weight (the reciprocal input)
                    const PlanarDst pd{dup2(p.x), dup2(p.y), dup2(p.z), dup2(wjr), dup2(wji), dup2(-wjr)};
                    const f2 nx = dup2(n.x), ny = dup2(n.y), nz = dup2(n.z);
                    f2 racc[3] = {0ull, 0ull, 0ull};
                    float2 *colw = &sCol[half * kSymWarps + warp][0];
                    float fr = 0.0f, fi = 0.0f;
                    for (int w = wA; w < nw; ++w) {
                        uint32_t m;
                        if (fl == kFlagBits) {
                            m = live ? a.mask.bits[(long long)(t * kWordsPerTile + w) * a.mask.pitch + j] : 0u;
                        } else {
                            const int nb = ntile - w * 32;
                            m = !live ? 0u : (nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u));
                        }
                        if (t == J) {
                            // diagonal tile: destination-owned, with the zero-input source limit
                            const int keep = limit - (i0 + w * 32);
                            m &= keep >= 32 ? 0xffffffffu : (keep <= 0 ? 0u : ((1u << keep) - 1u));
                            if (!__any_sync(0xffffffffu, m != 0u)) continue;
                            if (gate) diag_word<ATT, true>(a, sA, sB, w, m, d, fr, fi);
                            else diag_word<ATT, false>(a, sA, sB, w, m, d, fr, fi);
                            continue;
                        }
                        if (!__any_sync(0xffffffffu, m != 0u)) {
                            colw[w * 32 + lane] = make_float2(0.0f, 0.0f);
                            continue;
                        }
                        if (packed) {
                            if (gate) general_word<ATT, 2>(g, sA, sB, w, m, d, pd, nx, ny, nz, racc, colw, tr4, lane);
                            else if (__all_sync(0xffffffffu, m == 0xffffffffu))
                                general_word<ATT, 0>(g, sA, sB, w, m, d, pd, nx, ny, nz, racc, colw, tr4, lane);
                            else general_word<ATT, 1>(g, sA, sB, w, m, d, pd, nx, ny, nz, racc, colw, tr4, lane);
                        } else {
                            if (gate) sym_word<ATT, true>(a, sA, sB, w, m, d, wjr, wji, fr, fi, colw, tr2, lane);
                            else sym_word<ATT, false>(a, sA, sB, w, m, d, wjr, wji, fr, fi, colw, tr2, lane);
                        }
                    }
                    if (t < J)
                        for (int w = max(nw, wA); w < wB; ++w) colw[w * 32 + lane] = make_float2(0.0f, 0.0f);
                    if (packed) {
                        fr = flip * sum2(racc[0]);
                        fi = flip * (sum2(racc[1]) - sum2(racc[2]));
                    }
                    (half ? accr[1] : accr[0]) += (double)fr;
                    (half ? acci[1] : acci[0]) += (double)fi;
                }
                if (t < J) {
                    __syncthreads();
                    const double f = packed ? (double)flip : 1.0;
                    for (int s = wA * 32 + tid; s < wB * 32; s += kSymThreads) {
                        double sr = (double)sCol[0][s].x, si = (double)sCol[0][s].y;
#pragma unroll
                        for (int k = 1; k < 2 * kSymWarps; ++k) {
                            const float2 v = sCol[k][s];
                            sr += (double)v.x;
                            si += (double)v.y;
                        }
                        colpart[cbase + i0 + s] = make_double2(sr * f, si * f);
                    }
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
            rowpart[(long long)ch * kTile + q * kSymThreads + tid] = make_double2(accr[q], acci[q]);
    }
}

// P_out[cell] = rows + (P_in[i] != 0 ? columns : 0); P[cell] += P_out[cell].
// Rows: the general, then the planar chunks of the fragment's row in chunk
// order; columns: every non-empty block (I, J > I) of its tile I in J order
// (deterministic).  One CTA per tile, kFinSeg threads per fragment, each
// with a contiguous share of the chunks and of the J range; the shares are
// added in share order.  yrow / ycol: compressed-block rows and columns, may
// be null.
constexpr int kFinSeg = 4;
__global__ void __launch_bounds__(kFinSeg * kTile) k_finalize_f2f_sym(const double2 *rowpart, const int2 *chunk_off,
                                                                     const int *nchunks, int ndst,
                                                                     const double2 *colpart, const uint8_t *flags,
                                                                     int ntiles, const int *cell, const double2 *Pin,
                                                                     double2 *Pout, double2 *P, const double2 *yrow,
                                                                     const double2 *ycol)
{
    __shared__ double2 sR[kFinSeg - 1][kTile], sC[kFinSeg - 1][kTile];
    const int seg = threadIdx.x / kTile, f = threadIdx.x % kTile;
    const int I = blockIdx.x, q = I * kTile + f;
    double2 r = make_double2(0.0, 0.0), c = r;
    auto add = [](double2 &s, const double2 v) {
        s.x += v.x;
        s.y += v.y;
    };
    if (q < ndst) {
        const int2 c0 = chunk_off[I], c1 = chunk_off[I + 1];
        const int ng = c1.x - c0.x, n = ng + c1.y - c0.y, pbase = nchunks[1] + c0.y - ng;
        for (int k = n * seg / kFinSeg; k < n * (seg + 1) / kFinSeg; ++k)
            add(r, rowpart[(long long)(k < ng ? c0.x + k : pbase + k) * kTile + f]);
        // the tile's flag row, 16 flags at a time where aligned (rows of a
        // compressed bounce are mostly NONE)
        const uint8_t *frow = flags + (long long)I * ntiles;
        const int nJ = ntiles - (I + 1), Je = I + 1 + nJ * (seg + 1) / kFinSeg;
        for (int J = I + 1 + nJ * seg / kFinSeg; J < Je;) {
            if ((reinterpret_cast<uintptr_t>(frow + J) & 15u) == 0 && J + 16 <= Je) {
                const uint4 v = *reinterpret_cast<const uint4 *>(frow + J);
                if ((v.x | v.y | v.z | v.w) == 0u) {
                    J += 16;
                    continue;
                }
            }
            if (frow[J] != kFlagNone) add(c, colpart[(long long)kTile * J * (J - 1) / 2 + q]);
            ++J;
        }
    }
    if (seg > 0) {
        sR[seg - 1][f] = r;
        sC[seg - 1][f] = c;
    }
    __syncthreads();
    if (seg > 0 || q >= ndst) return;
#pragma unroll
    for (int s = 0; s < kFinSeg - 1; ++s) {
        add(r, sR[s][f]);
        add(c, sC[s][f]);
    }
    double sr = r.x, si = r.y;
    const int cl = cell[q];
    const double2 pin = Pin[cl];
    if (yrow) {
        sr += yrow[q].x;
        si += yrow[q].y;
    }
    if (pin.x != 0.0 || pin.y != 0.0) {
        sr += c.x;
        si += c.y;
        if (ycol) {
            sr += ycol[q].x;
            si += ycol[q].y;
        }
    }
    Pout[cl] = make_double2(sr, si);
    double2 o = P[cl];
    o.x += sr;
    o.y += si;
    P[cl] = o;
}

}  // namespace

// Chunk shape by problem size.  Blocks: about ntiles^2 / 2.  Planar chunks grow
// with the problem (their row partials, 4 KB a chunk, are written and read
// again) while some 16 of them are left per resident CTA, so that the last
// ones do not leave the GPU idle; general blocks cost twice as much and are
// few where planar ones are many, one to a chunk (the 60 kHz compressed
// remainder, 3.4k blocks: two to a chunk 0.48 ms, one 0.45).  With fewer than
// 4 blocks per CTA the blocks themselves are cut into word ranges (190 blocks
// of a 20-tile plate pair: 0.23 ms uncut, 0.05 ms in eighths).
SymShape sym_shape(int ntiles, int nsm)
{
    const long long blocks = (long long)ntiles * (ntiles + 1) / 2, slots = 4LL * std::max(nsm, 1);
    SymShape s;
    s.per_planar = (int)std::min<long long>(4, std::max<long long>(1, blocks / (16 * slots)));
    s.per_general = 1;
    s.sub = 1;
    while (s.sub < kWordsPerTile && blocks * s.sub < 4 * slots) s.sub *= 2;
    return s;
}

// Chunks that there is room for (4 KB of row partials each): all that the shape
// can make, or, in problems of more than kSymChunks, what two blocks to a chunk
// can: one to a chunk would take 31 GB at a million fragments instead of 16,
// and most of it would not be written (in large problems nearly all blocks are
// planar, up to four to a chunk, or empty).  k_sym_scan falls back to two where
// the chunks do not fit.
constexpr size_t kSymChunks = 1 << 14;
size_t sym_max_chunks(int ntiles, const SymShape &s)
{
    size_t all = 0, paired = 0;
    for (int J = 0; J < ntiles; J++) {
        all += s.sub > 1 ? (size_t)(J + 1) * s.sub : (size_t)(J + 1);
        // g general and p planar blocks: (g + 1) / 2 + (p + 1) / 2 <= (g + p) / 2 + 1
        paired += (size_t)(J + 1) / 2 + 1;
    }
    return s.sub > 1 ? all : std::min(all, std::max(paired, kSymChunks));
}

namespace {
// the packed forms divide by k / (4 pi)
int packed_ok(const SumArgs &a)
{
    return a.geom && a.kr4pi > 1e-12f && a.kr4pi < 1e12f && a.ka <= 1e6f * a.kr;
}
}  // namespace

void launch_sym_worklist(const SumArgs &a, const SymShape &sh, size_t max_chunks, int *blist, int2 *rowcnt,
                         int2 *chunk_off, int4 *chunks, int *nchunks, cudaStream_t s)
{
    const int nb = a.mask.ndstblocks, ntiles = a.mask.ntiles;
    if (nb <= 0) return;
    k_sym_rows<<<nb, kTile, 0, s>>>(a, ntiles, nb, packed_ok(a), blist, rowcnt);
    k_sym_scan<<<1, 1024, 0, s>>>(rowcnt, nb, sh, (int)std::min<size_t>(max_chunks, INT_MAX), chunk_off, nchunks);
    k_sym_fill<<<nb, 128, 0, s>>>(rowcnt, chunk_off, nchunks, sh.sub, chunks);
}

void launch_sum_f2f_sym(const SumArgs &a, SymWork wl, int nsm, double2 *colpart, double2 *rowpart, cudaStream_t s)
{
    if (a.nsrc <= 0 || a.ndst <= 0) return;
    wl.packed_ok = packed_ok(a);
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(k_sum_f2f_sym<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSymDynSmem);
        cudaFuncSetAttribute(k_sum_f2f_sym<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSymDynSmem);
        attr_set = true;
    }
    const unsigned grid = 4u * (unsigned)std::max(nsm, 1);
    if (a.ka != 0.0f)
        k_sum_f2f_sym<true><<<grid, kSymThreads, kSymDynSmem, s>>>(a, wl, colpart, rowpart);
    else
        k_sum_f2f_sym<false><<<grid, kSymThreads, kSymDynSmem, s>>>(a, wl, colpart, rowpart);
}

void launch_finalize_f2f_sym(const double2 *rowpart, const int2 *chunk_off, const int *nchunks, int ndst,
                             const double2 *colpart, const uint8_t *flags, int ntiles, const int *cell,
                             const double2 *Pin, double2 *Pout, double2 *P, cudaStream_t s, const double2 *yrow,
                             const double2 *ycol)
{
    if (ndst > 0)
        k_finalize_f2f_sym<<<(unsigned)((ndst + kTile - 1) / kTile), kFinSeg * kTile, 0, s>>>(
            rowpart, chunk_off, nchunks, ndst, colpart, flags, ntiles, cell, Pin, Pout, P, yrow, ycol);
}

}  // namespace sonar
