// sums.cu -- destination-owned sums: source points -> cells, fragments ->
// field points, target -> field object, target -> target, and the ordered
// form of the bounce sum (OptiX.cu:35-190, :192-406).
//
// A CTA owns 256 destinations and a range of 256-source tiles; each tile's
// data are staged in shared memory and read as warp broadcasts.  No atomics:
// partial sums per source split are reduced in a fixed order.
//
// The readout and the two target -> other-object hops run packed: two sources
// to a register (pack2.cuh), and, where a tile lies on one facet, the
// fragment's cosine as the destination's distance from the tile's plane, taken
// out of the pair loop.  The distance keeps the reference's FP32 rounding
// (|v|^2 without contraction, r rounded), as the scalar form's: at 30 m the
// rounding of r is 3e-4 rad of phase at 40 kHz and parity is defined by it.
// The source hop (a handful of sources), centroid-relative geometry and the
// ordered bounce sum run the scalar pair arithmetic.
//
// What bounds the packed form: FP32 lanes, 26 operations a pair on a one-facet
// tile (30 otherwise) against 32 lanes per clock and scheduler, beside 3
// special-function operations at 4 lanes; the scalar form took about 42 issue
// slots.  Trihedral at 40 kHz onto 65,536 points (3.0e9 pairs in blocks that
// interact, one-facet tiles): 4.37 -> 2.79 ms; icosphere at 20 kHz onto 512 x 512
// cells (7 facets to a tile): 17.1 -> 10.3 ms; plate at 10 kHz onto 4,096 points,
// 6 tiles in eighths: 0.053 -> 0.016 ms.
#include "sonar_internal.h"
#include "green.cuh"
#include "pack2.cuh"

#include <algorithm>

namespace sonar {
namespace {

// One pair's term.  GATE: also evaluate the pair's cosine gates inline (CLEAR
// blocks) and return them in ok.
template <int HOP, bool ATT, bool GATE>
__device__ __forceinline__ void pair_term(const SumArgs &a, const float4 A, const float4 B, const Dst &d, float &tr,
                                          float &ti, bool &ok)
{
    // v = p_dst - p_src; |v|^2 with the reference's rounding (its r feeds the phase)
    const float vx = __fsub_rn(d.px, A.x), vy = __fsub_rn(d.py, A.y), vz = __fsub_rn(d.pz, A.z);
    const float r2 = dot_rn(vx, vy, vz, vx, vy, vz);
    // r: one Newton step on the reciprocal square root, r = r0 + (r2 - r0^2) / (2 r0)
    // with r0 = r2 * rsqrt(r2); within an ulp of the correctly rounded root
    const float rinv = rsqrtf(r2);
    const float r0 = r2 * rinv;
    const float r = fmaf(fmaf(-r0, r0, r2), 0.5f * rinv, r0);
    // phase k r in turns: r * (k / 2 pi) as an exact two-float product plus the
    // low part of k / 2 pi, the integer part removed exactly
    const float th = __fmul_rn(r, a.k2hi);
    const float tl = fmaf(r, a.k2lo, fmaf(r, a.k2hi, -th));
    const float frac = (th - rintf(th)) + tl;
    float sn, cs;
    __sincosf(frac * kTwoPi, &sn, &cs);
    const float damp = ATT ? __expf(-a.ka * r) : 1.0f;
    ok = true;
    if (HOP == HOP_SRC) {
        // cos_inc P e^{ikr} / r
        float ci = -(vx * d.nx + vy * d.ny + vz * d.nz) * rinv;
        if (a.dst_is_field)
            ci = 1.0f;
        else if (GATE)
            ok = gate_from(ci, vx, vy, vz, -1.0f, d.nx, d.ny, d.nz);
        const float amp = ATT ? ci * rinv * damp : ci * rinv;
        const float er = amp * cs, ei = amp * sn;
        tr = er * A.w - ei * B.w;
        ti = er * B.w + ei * A.w;
    } else {
        // -e^{ikr}/(4 pi) * (ik/r) + 1/r^2
        const float rinv2 = rinv * rinv;
        float gr, gi;
        if (ATT) {
            const float amp = rinv * kInv4Pi * damp;
            gr = fmaf(amp, fmaf(a.ka, cs, a.kr * sn), rinv2);
            gi = amp * fmaf(a.ka, sn, -a.kr * cs);
        } else {
            const float ampk = rinv * (kInv4Pi * a.kr);
            gr = fmaf(ampk, sn, rinv2);
            gi = -ampk * cs;
        }
        const float c1 = (vx * B.x + vy * B.y + vz * B.z) * rinv;  // cos_scat (source side)
        float wgt;
        if (HOP == HOP_F2F || HOP == HOP_RESP) {
            const float c2 = -(vx * d.nx + vy * d.ny + vz * d.nz) * rinv;  // cos_inc (destination side)
            wgt = c1 * c2;
            if (GATE) ok = gate_from(c1, vx, vy, vz, 1.0f, B.x, B.y, B.z) && gate_from(c2, vx, vy, vz, -1.0f, d.nx, d.ny, d.nz);
        } else {
            wgt = c1;
            if (GATE) ok = gate_from(c1, vx, vy, vz, 1.0f, B.x, B.y, B.z);
        }
        if (HOP != HOP_FP) {
            // regularised G below r_min = delta_src (OptiX.cu:340-346); near the
            // threshold the branch uses the correctly rounded r, as the reference
            float rr = r;
            if (fabsf(r - a.rmin) <= a.rmin * 4e-7f) rr = __fsqrt_rn(r2);
            if (rr < a.rmin) {
                gr = -a.ka * kInv4Pi;
                gi = a.kr * kInv4Pi;
            }
        }
        gr *= wgt;
        gi *= wgt;
        tr = gr * A.w - gi * B.w;
        ti = gr * B.w + gi * A.w;
    }
}

// pair_term of the source hop and the readout with the phase distance taken
// relative to an FP64 reference (o: the fragment's offset from its tile
// centroid for the readout).  The source hop evaluates its distance in FP64
// outright: it has S x N_cells pairs, a few per fragment.
struct RelRef;
template <int HOP, bool ATT>
__device__ __forceinline__ void pair_term_rel(const SumArgs &a, const float4 A, const float4 B, const Dst &d,
                                              const RelRef &ref, float4 o, bool gate, float &tr, float &ti, bool &ok);

// Phase of a pair in turns from a distance known in FP64 to within FP32
// round-off of a small correction: r = R + dr, R (FP64) the distance to a
// reference point, phase0 = frac(R k / 2 pi) reduced in FP64 once, dr in FP32.
__device__ __forceinline__ float rel_turns(float phase0, float dr, const SumArgs &a)
{
    const float th = __fmul_rn(dr, a.k2hi);
    const float tl = fmaf(dr, a.k2lo, fmaf(dr, a.k2hi, -th));
    const float f = phase0 + ((th - rintf(th)) + tl);
    return f - rintf(f);
}

// Relative geometry of the readout (HOP_FP): with o = p_i - c (fragment from
// its tile's centroid, small) and D = p_j - c (field point from the centroid,
// R = |D| in FP64), r^2 = R^2 - 2 o.D + |o|^2, so r - R = (|o|^2 - 2 o.D) /
// (r + R): FP32 arithmetic on small numbers, no cancellation at large R.
struct RelRef {
    float dx, dy, dz, R, phase0;
};

__device__ __forceinline__ RelRef rel_ref(const SumArgs &a, double px, double py, double pz, float4 c)
{
    const double dx = px - (double)c.x, dy = py - (double)c.y, dz = pz - (double)c.z;
    const double R = sqrt(dx * dx + dy * dy + dz * dz);
    const double t = R * a.k2pi;
    return RelRef{(float)dx, (float)dy, (float)dz, (float)R, (float)(t - floor(t))};
}

template <int HOP, bool ATT>
__device__ __forceinline__ void pair_term_rel(const SumArgs &a, const float4 A, const float4 B, const Dst &d,
                                              const RelRef &ref, float4 o, bool gate, float &tr, float &ti, bool &ok)
{
    // direction, cosines and amplitudes from the FP32 difference (relative
    // accuracy ~1e-7 is enough for them); only the phase needs r to ~1e-9 m
    const float vx = __fsub_rn(d.px, A.x), vy = __fsub_rn(d.py, A.y), vz = __fsub_rn(d.pz, A.z);
    const float r2 = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
    const float rinv = rsqrtf(r2);
    const float r = r2 * rinv;
    float turns;
    if (HOP == HOP_SRC) {
        const double ex = (double)d.px - (double)A.x, ey = (double)d.py - (double)A.y, ez = (double)d.pz - (double)A.z;
        const double t = sqrt(ex * ex + ey * ey + ez * ez) * a.k2pi;
        turns = (float)(t - rint(t));
    } else {
        // r - R = (|o|^2 - 2 o.D) / (r + R)
        const float num = fmaf(-2.0f, fmaf(o.x, ref.dx, fmaf(o.y, ref.dy, o.z * ref.dz)), o.w);
        turns = rel_turns(ref.phase0, num / (r + ref.R), a);
    }
    float sn, cs;
    __sincosf(turns * kTwoPi, &sn, &cs);
    const float damp = ATT ? __expf(-a.ka * r) : 1.0f;
    ok = true;
    if (HOP == HOP_SRC) {
        float ci = -(vx * d.nx + vy * d.ny + vz * d.nz) * rinv;
        if (a.dst_is_field)
            ci = 1.0f;
        else if (gate)
            ok = gate_from(ci, vx, vy, vz, -1.0f, d.nx, d.ny, d.nz);
        const float amp = ATT ? ci * rinv * damp : ci * rinv;
        const float er = amp * cs, ei = amp * sn;
        tr = er * A.w - ei * B.w;
        ti = er * B.w + ei * A.w;
    } else {
        const float rinv2 = rinv * rinv;
        float gr, gi;
        if (ATT) {
            const float amp = rinv * kInv4Pi * damp;
            gr = fmaf(amp, fmaf(a.ka, cs, a.kr * sn), rinv2);
            gi = amp * fmaf(a.ka, sn, -a.kr * cs);
        } else {
            const float ampk = rinv * (kInv4Pi * a.kr);
            gr = fmaf(ampk, sn, rinv2);
            gi = -ampk * cs;
        }
        const float c1 = (vx * B.x + vy * B.y + vz * B.z) * rinv;  // cos_scat
        if (gate) ok = gate_from(c1, vx, vy, vz, 1.0f, B.x, B.y, B.z);
        gr *= c1;
        gi *= c1;
        tr = gr * A.w - gi * B.w;
        ti = gr * B.w + gi * A.w;
    }
}

// The scalar form: the source hop, centroid-relative geometry, the ordered
// bounce sum.
template <int HOP, bool ATT, bool REL = false>
__global__ void __launch_bounds__(kTile) k_sum(SumArgs a)
{
    __shared__ float4 sA[kTile];
    __shared__ float4 sB[kTile];
    __shared__ float4 sO[REL && HOP == HOP_FP ? kTile : 1];  // fragment offsets from the tile centroid
    const int tid = threadIdx.x;
    const int j = blockIdx.x * kTile + tid;
    const bool live = j < a.ndst;
    Dst d{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    int limit = a.nsrc;
    if (live) {
        const float4 p = a.dst_pos[j];
        d.px = p.x; d.py = p.y; d.pz = p.z;
        if (a.dst_facet) {
            const float4 n = a.dst_facet_n[a.dst_facet[j]];
            d.nx = n.x; d.ny = n.y; d.nz = n.z;
        }
        if (HOP == HOP_F2F) limit = a.dst_limit[j];
    }
    double accr = 0.0, acci = 0.0;
    const int t0 = blockIdx.y * a.tiles_per_split;
    const int t1 = min(t0 + a.tiles_per_split, a.mask.ntiles);
    for (int t = t0; t < t1; ++t) {
        const uint8_t fl = a.mask.flags[(long long)t * a.mask.ndstblocks + blockIdx.x];  // uniform per CTA
        if (fl == kFlagNone) continue;
        __syncthreads();
        RelRef ref{};
        {
            const int i = t * kTile + tid;
            const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            sA[tid] = i < a.nsrc ? a.srcA[i] : z;
            sB[tid] = i < a.nsrc ? a.srcB[i] : z;
            if (REL && HOP == HOP_FP) {
                const float4 c = a.tile_cen[t];
                const float4 p = sA[tid];
                const float ox = p.x - c.x, oy = p.y - c.y, oz = p.z - c.z;
                sO[tid] = make_float4(ox, oy, oz, fmaf(ox, ox, fmaf(oy, oy, oz * oz)));
                ref = rel_ref(a, (double)d.px, (double)d.py, (double)d.pz, c);
            }
        }
        __syncthreads();
        const int ntile = min(kTile, a.nsrc - t * kTile);
        const int nw = (ntile + 31) >> 5;
        float fr = 0.0f, fi = 0.0f;
        for (int w = 0; w < nw; ++w) {
            uint32_t m;
            if (fl == kFlagBits) {
                m = live ? a.mask.bits[(long long)(t * kWordsPerTile + w) * a.mask.pitch + j] : 0u;
            } else {
                const int nb = ntile - w * 32;  // CLEAR / ALL: every valid source
                m = !live ? 0u : (nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u));
            }
            if (HOP == HOP_F2F) {
                // FACET_SELF zero-input rule: when this destination's input is 0
                // the sources of higher facets (its reciprocal partners) drop out
                const int keep = limit - (t * kTile + w * 32);
                m &= keep >= 32 ? 0xffffffffu : (keep <= 0 ? 0u : ((1u << keep) - 1u));
            }
            if (!__any_sync(0xffffffffu, m != 0u)) continue;
            const int bmax = min(32, ntile - w * 32);  // a source hop often has a handful of sources
            if (REL) {
                // centroid-relative phase (the gates of CLEAR blocks inline as below)
#pragma unroll 4
                for (int b = 0; b < bmax; ++b) {
                    const float4 A = sA[w * 32 + b];
                    const float4 B = sB[w * 32 + b];
                    float tr, ti;
                    bool ok;
                    pair_term_rel<HOP, ATT>(a, A, B, d, ref, REL && HOP == HOP_FP ? sO[w * 32 + b] : A,
                                            fl == kFlagClear, tr, ti, ok);
                    const bool on = ((m >> b) & 1u) && ok;
                    fr += on ? tr : 0.0f;
                    fi += on ? ti : 0.0f;
                }
            } else if (fl != kFlagClear) {
#pragma unroll 4
                for (int b = 0; b < bmax; ++b) {
                    const float4 A = sA[w * 32 + b];
                    const float4 B = sB[w * 32 + b];
                    float tr, ti;
                    bool ok;
                    pair_term<HOP, ATT, false>(a, A, B, d, tr, ti, ok);
                    const bool on = (m >> b) & 1u;
                    fr += on ? tr : 0.0f;
                    fi += on ? ti : 0.0f;
                }
            } else {
#pragma unroll 4
                for (int b = 0; b < bmax; ++b) {
                    const float4 A = sA[w * 32 + b];
                    const float4 B = sB[w * 32 + b];
                    float tr, ti;
                    bool ok;
                    pair_term<HOP, ATT, true>(a, A, B, d, tr, ti, ok);
                    const bool on = ((m >> b) & 1u) && ok;
                    fr += on ? tr : 0.0f;
                    fi += on ? ti : 0.0f;
                }
            }
        }
        accr += (double)fr;
        acci += (double)fi;
    }
    if (live) a.partial[(long long)blockIdx.y * a.ndst + j] = make_double2(accr, acci);
}

// ---------------------------------------------------------------- packed sums
// Constants of a packed pair loop.
struct Pair2 {
    Phase2 ph;
    f2 half, c4pik, natt, qatt, nqatt;
};
__device__ __forceinline__ Pair2 pair2(const SumArgs &a)
{
    return Pair2{phase2(a.k2hi, a.k2lo), dup2(0.5f), dup2(1.0f / a.kr4pi), dup2(-a.ka * 1.44269504088896341f),
                 dup2(a.ka / a.kr), dup2(-(a.ka / a.kr))};
}

// One destination against one 32-source word.  sA: source pairs (x0 x1 y0
// y1) and, 128 entries on, (z0 z1 wr0 wr1); sB: (wi0 wi1 nz0 nz1) and (nx0 nx1
// ny0 ny1).  The pair's term is (4 pi / k) G times the source's cosine (UNI:
// without the plane distance, which the caller has) and, for HOP_RESP, minus
// the destination's.  MODE 0: every pair; 1: the pairs of m.
// acc: Re, and the two parts of Im.
template <int HOP, bool ATT, bool UNI, int MODE>
__device__ __forceinline__ void sum_word(const Pair2 &g, const float4 *sA, const float4 *sB, int w, uint32_t m, f2 px,
                                         f2 py, f2 pz, f2 nx, f2 ny, f2 nz, f2 (&acc)[3])
{
#pragma unroll 4
    for (int b = 0; b < 16; ++b) {
        const int q = w * 16 + b;
        const ulonglong2 XY = *reinterpret_cast<const ulonglong2 *>(&sA[q]);
        const ulonglong2 ZW = *reinterpret_cast<const ulonglong2 *>(&sA[kTile / 2 + q]);
        const f2 vx = sub2(px, XY.x), vy = sub2(py, XY.y), vz = sub2(pz, ZW.x);
        f2 WI, d1 = 0ull;
        if (UNI) {
            WI = *reinterpret_cast<const f2 *>(&sB[q]);
        } else {
            const ulonglong2 IN = *reinterpret_cast<const ulonglong2 *>(&sB[q]);
            const ulonglong2 NN = *reinterpret_cast<const ulonglong2 *>(&sB[kTile / 2 + q]);
            WI = IN.x;
            d1 = fma2(vx, NN.x, fma2(vy, NN.y, mul2(vz, IN.y)));  // r cos_scat
        }
        // the reference's FP32 |v|^2 and r (Newton step on rsqrt, within an ulp
        // of the rounded root)
        const f2 r2 = dot_rn2(vx, vy, vz);
        const f2 rinv = rsqrt2(r2);
        const f2 r0 = mul2(r2, rinv);
        const f2 r = fma2(fma2(r0 ^ 0x8000000080000000ull, r0, r2), mul2(rinv, g.half), r0);
        f2 f = fma2(r, g.ph.khi, sub2(g.ph.magic, fma2(r, g.ph.khi, g.ph.magic)));
        f = mul2(fma2(r, g.ph.klo, f), g.ph.two_pi);
        float f0, f1, s0, c0, s1, c1;
        up2(f, f0, f1);
        __sincosf(f0, &s0, &c0);
        __sincosf(f1, &s1, &c1);
        const f2 sn = pk2(s0, s1), cs = pk2(c0, c1);
        f2 amp = mul2(rinv, rinv);
        if (HOP == HOP_RESP) amp = mul2(mul2(amp, rinv), fma2(vx, nx, fma2(vy, ny, mul2(vz, nz))));
        if (!UNI) amp = mul2(amp, d1);
        f2 Tr, Ti;
        if (ATT) {
            const f2 osc = mul2(amp, ex2_2(mul2(r, g.natt)));
            Tr = fma2(osc, fma2(g.qatt, cs, sn), mul2(amp, mul2(rinv, g.c4pik)));
            Ti = mul2(osc, fma2(g.nqatt, sn, cs));
        } else {
            Tr = mul2(amp, fma2(rinv, g.c4pik, sn));
            Ti = mul2(amp, cs);
        }
        if (MODE > 0) {
            const bool on0 = (m >> (2 * b)) & 1u, on1 = (m >> (2 * b + 1)) & 1u;
            float a0, a1, b0, b1;
            up2(Tr, a0, a1);
            up2(Ti, b0, b1);
            Tr = pk2(on0 ? a0 : 0.0f, on1 ? a1 : 0.0f);
            Ti = pk2(on0 ? b0 : 0.0f, on1 ? b1 : 0.0f);
        }
        // T w with T = Tr - i Ti
        acc[0] = fma2(Tr, ZW.y, fma2(Ti, WI, acc[0]));
        acc[1] = fma2(Tr, WI, acc[1]);
        acc[2] = fma2(Ti, ZW.y, acc[2]);
    }
}

// The packed form: grid (destination blocks, tile splits, word splits); word
// split z of wsplit takes its share of every tile's words (few-tile problems).
// A tile takes the scalar pair loop where the packed one does not apply: pairs
// that can reach r_min (or coincide), coordinates beyond 1e6, a vanishing k,
// weights (or distances) whose terms would leave FP32, and gates to evaluate
// (CLEAR) that the plane distance does not decide.
template <int HOP, bool ATT>
__global__ void __launch_bounds__(kTile, 3) k_sum_packed(SumArgs a)
{
    __shared__ float4 sA[kTile], sB[kTile];
    __shared__ int sBox[6];
    const int tid = threadIdx.x, lane = tid & 31;
    const int j = blockIdx.x * kTile + tid;
    const bool live = j < a.ndst;
    const float4 p = a.dst_pos[live ? j : blockIdx.x * kTile];
    float4 n = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (HOP == HOP_RESP) n = a.dst_facet_n[a.dst_facet[live ? j : blockIdx.x * kTile]];
    const Dst d{p.x, p.y, p.z, n.x, n.y, n.z};
    // box of the destinations
    if (tid < 6) sBox[tid] = tid < 3 ? f2o(3.0e38f) : f2o(-3.0e38f);
    __syncthreads();
    {
        const float c[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int lo = __reduce_min_sync(0xffffffffu, f2o(c[k])), hi = __reduce_max_sync(0xffffffffu, f2o(c[k]));
            if (lane == 0) {
                atomicMin(&sBox[k], lo);
                atomicMax(&sBox[3 + k], hi);
            }
        }
    }
    __syncthreads();
    const float4 blo = make_float4(o2f(sBox[0]), o2f(sBox[1]), o2f(sBox[2]), 0.0f);
    const float4 bhi = make_float4(o2f(sBox[3]), o2f(sBox[4]), o2f(sBox[5]), 0.0f);
    const Pair2 g = pair2(a);
    const f2 px = dup2(p.x), py = dup2(p.y), pz = dup2(p.z);
    const f2 nx = dup2(n.x), ny = dup2(n.y), nz = dup2(n.z);
    const bool k_ok = a.kr4pi > 1e-12f && a.kr4pi < 1e12f && a.ka <= 1e6f * a.kr;
    double accr = 0.0, acci = 0.0;
    const int t0 = blockIdx.y * a.tiles_per_split;
    const int t1 = min(t0 + a.tiles_per_split, a.mask.ntiles);
    const int words = kWordsPerTile / a.wsplit, w0 = blockIdx.z * words;
    for (int t = t0; t < t1; ++t) {
        const uint8_t fl = a.mask.flags[(long long)t * a.mask.ndstblocks + blockIdx.x];  // uniform per CTA
        if (fl == kFlagNone) continue;
        const TileGeom gt = a.geom[t];
        const bool uni = gt.n.w != 0.0f;
        const float rfar = HOP == HOP_FP ? 1e-9f : fmaxf(a.rmin * 1.001f, 1e-9f);
        const float gap = box_gap(gt.lo, gt.hi, blo, bhi);
        bool packed = k_ok && gap > rfar && fmaxf(box_extent(gt.lo, gt.hi), box_extent(blo, bhi)) < 1e6f &&
                      packed_in_range(a, gap, box_diag(gt.lo, gt.hi, blo, bhi), gt.wmax);
        // CLEAR: with one facet the plane distance decides a destination's gate
        // for the whole tile outside the margin of FP32 rounding; the
        // destination's own cosine (HOP_RESP) is left to the scalar form
        float d1 = 0.0f;
        bool off = false;
        if (uni) d1 = plane_distance(gt, p.x, p.y, p.z);
        if (fl == kFlagClear) {
            const float rx = fmaxf(fabsf(p.x - gt.lo.x), fabsf(p.x - gt.hi.x)),
                        ry = fmaxf(fabsf(p.y - gt.lo.y), fabsf(p.y - gt.hi.y)),
                        rz = fmaxf(fabsf(p.z - gt.lo.z), fabsf(p.z - gt.hi.z));
            const float rmax = 1.0001f * sqrtf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
            const float margin = 1e-6f * (5.0f * rmax + fabsf(p.x) + fabsf(p.y) + fabsf(p.z) +
                                          3.0f * box_extent(gt.lo, gt.hi));
            off = d1 < -margin;
            const bool sure = HOP != HOP_RESP && uni && fabsf(d1) > margin;
            packed = packed && __syncthreads_and(sure);
        }
        __syncthreads();
        const int i0 = t * kTile;
        {
            // thread tid stages source tid of the scalar layout, threads below 128
            // a source pair of the packed one
            if (packed) {
                if (tid < kTile / 2) {
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
                    sA[kTile / 2 + tid] = make_float4(A[0].z, A[1].z, A[0].w, A[1].w);
                    sB[tid] = make_float4(B[0].w, B[1].w, B[0].z, B[1].z);
                    sB[kTile / 2 + tid] = make_float4(B[0].x, B[1].x, B[0].y, B[1].y);
                }
            } else {
                const int i = i0 + tid;
                const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                sA[tid] = i < a.nsrc ? a.srcA[i] : z;
                sB[tid] = i < a.nsrc ? a.srcB[i] : z;
            }
            __syncthreads();
        }
        const int ntile = min(kTile, a.nsrc - i0);
        const int w1 = min((ntile + 31) >> 5, w0 + words);
        f2 acc[3] = {0ull, 0ull, 0ull};
        float fr = 0.0f, fi = 0.0f;
        for (int w = w0; w < w1; ++w) {
            uint32_t m;
            if (fl == kFlagBits) {
                m = live ? a.mask.bits[(long long)(t * kWordsPerTile + w) * a.mask.pitch + j] : 0u;
            } else {
                const int nb = ntile - w * 32;  // CLEAR / ALL: every valid source
                m = !live ? 0u : (nb >= 32 ? 0xffffffffu : ((1u << nb) - 1u));
            }
            if (off) m = 0u;
            if (!__any_sync(0xffffffffu, m != 0u)) continue;
            if (packed) {
                // padded sources carry no weight, dead threads write nothing
                const bool all = fl == kFlagAll || __all_sync(0xffffffffu, m == 0xffffffffu || !live);
                if (uni) {
                    if (all) sum_word<HOP, ATT, true, 0>(g, sA, sB, w, m, px, py, pz, nx, ny, nz, acc);
                    else sum_word<HOP, ATT, true, 1>(g, sA, sB, w, m, px, py, pz, nx, ny, nz, acc);
                } else {
                    if (all) sum_word<HOP, ATT, false, 0>(g, sA, sB, w, m, px, py, pz, nx, ny, nz, acc);
                    else sum_word<HOP, ATT, false, 1>(g, sA, sB, w, m, px, py, pz, nx, ny, nz, acc);
                }
            } else {
                const int bmax = min(32, ntile - w * 32);
#pragma unroll 2
                for (int b = 0; b < bmax; ++b) {
                    const float4 A = sA[w * 32 + b];
                    const float4 B = sB[w * 32 + b];
                    float tr, ti;
                    bool ok;
                    pair_term<HOP, ATT, true>(a, A, B, d, tr, ti, ok);
                    const bool on = ((m >> b) & 1u) && (ok || fl != kFlagClear);
                    fr += on ? tr : 0.0f;
                    fi += on ? ti : 0.0f;
                }
            }
        }
        if (packed) {
            float s = HOP == HOP_RESP ? -a.kr4pi : a.kr4pi;
            if (uni) s *= d1;
            fr = off ? 0.0f : s * sum2(acc[0]);
            fi = off ? 0.0f : s * (sum2(acc[1]) - sum2(acc[2]));
        }
        accr += (double)fr;
        acci += (double)fi;
    }
    if (live) a.partial[(long long)(blockIdx.y * a.wsplit + blockIdx.z) * a.ndst + j] = make_double2(accr, acci);
}

// ---------------------------------------------------------------- finalize
// The splits' partial sums of each destination, added in SHARES contiguous
// shares of the splits (the shares then in order), into
//   FIN_ADD   out[cell] += s
//   FIN_F2F   P_out[cell] = s, out[cell] += s
//   FIN_RESP  P_out[cell] += s, out[cell] += s; with gate_pin, destinations
//             whose P_in is 0 receive nothing (the zero-input skip of the
//             first object's cell also kills its reciprocal term,
//             OptiX.cu:241-245, :367-390)
// A thread that reads its splits one after the other is bound by that chain
// (19 us for 69 splits of 4,096 points): many splits take eight threads.
constexpr int FIN_ADD = 0, FIN_F2F = 1, FIN_RESP = 2;
template <int MODE, int SHARES>
__global__ void __launch_bounds__(kTile) k_finalize(const double2 *partial, int nsplit, int ndst, const int *cell,
                                                   const double2 *gate_pin, double2 *Pout, double2 *out)
{
    constexpr int kDst = kTile / SHARES;
    __shared__ double2 sS[SHARES][kDst];
    const int l = threadIdx.x % kDst, g = threadIdx.x / kDst;
    const int j = blockIdx.x * kDst + l;
    double sr = 0.0, si = 0.0;
    if (j < ndst)
        for (int k = nsplit * g / SHARES; k < nsplit * (g + 1) / SHARES; ++k) {
            const double2 v = partial[(long long)k * ndst + j];
            sr += v.x;
            si += v.y;
        }
    if (SHARES > 1) {
        sS[g][l] = make_double2(sr, si);
        __syncthreads();
    }
    if (g > 0 || j >= ndst) return;
    const int c = cell ? cell[j] : j;
    if (MODE == FIN_RESP && gate_pin) {
        const double2 p = gate_pin[c];
        if (p.x == 0.0 && p.y == 0.0) return;
    }
#pragma unroll
    for (int k = 1; k < SHARES; ++k) {
        sr += sS[k][l].x;
        si += sS[k][l].y;
    }
    double2 o;
    if (MODE == FIN_F2F) Pout[c] = make_double2(sr, si);
    if (MODE == FIN_RESP) {
        o = Pout[c];
        o.x += sr;
        o.y += si;
        Pout[c] = o;
    }
    o = out[c];
    o.x += sr;
    o.y += si;
    out[c] = o;
}

template <int MODE>
void finalize(const double2 *partial, int nsplit, int ndst, const int *cell, const double2 *gate_pin, double2 *Pout,
              double2 *out, cudaStream_t s)
{
    if (ndst <= 0) return;
    if (nsplit >= 16)
        k_finalize<MODE, 8><<<(unsigned)((ndst + 31) / 32), kTile, 0, s>>>(partial, nsplit, ndst, cell, gate_pin, Pout,
                                                                           out);
    else
        k_finalize<MODE, 1><<<(unsigned)((ndst + kTile - 1) / kTile), kTile, 0, s>>>(partial, nsplit, ndst, cell,
                                                                                     gate_pin, Pout, out);
}

}  // namespace

void launch_sum(const SumArgs &a, cudaStream_t s)
{
    if (a.nsrc <= 0 || a.ndst <= 0) return;
    const dim3 grid(a.mask.ndstblocks, a.nsplit), pgrid(a.mask.ndstblocks, a.nsplit / a.wsplit, a.wsplit);
    const bool att = a.ka != 0.0f;
    switch (a.hop) {
    case HOP_SRC:
        if (a.rel) {
            if (att) k_sum<HOP_SRC, true, true><<<grid, kTile, 0, s>>>(a);
            else k_sum<HOP_SRC, false, true><<<grid, kTile, 0, s>>>(a);
        } else {
            if (att) k_sum<HOP_SRC, true><<<grid, kTile, 0, s>>>(a);
            else k_sum<HOP_SRC, false><<<grid, kTile, 0, s>>>(a);
        }
        break;
    case HOP_FP:
        if (a.rel) {
            if (att) k_sum<HOP_FP, true, true><<<grid, kTile, 0, s>>>(a);
            else k_sum<HOP_FP, false, true><<<grid, kTile, 0, s>>>(a);
        } else {
            if (att) k_sum_packed<HOP_FP, true><<<pgrid, kTile, 0, s>>>(a);
            else k_sum_packed<HOP_FP, false><<<pgrid, kTile, 0, s>>>(a);
        }
        break;
    case HOP_F2F:
        if (att) k_sum<HOP_F2F, true><<<grid, kTile, 0, s>>>(a);
        else k_sum<HOP_F2F, false><<<grid, kTile, 0, s>>>(a);
        break;
    case HOP_RESP:
        if (att) k_sum_packed<HOP_RESP, true><<<pgrid, kTile, 0, s>>>(a);
        else k_sum_packed<HOP_RESP, false><<<pgrid, kTile, 0, s>>>(a);
        break;
    default:
        if (att) k_sum_packed<HOP_NORESP, true><<<pgrid, kTile, 0, s>>>(a);
        else k_sum_packed<HOP_NORESP, false><<<pgrid, kTile, 0, s>>>(a);
        break;
    }
}

void launch_finalize_add(const double2 *partial, int nsplit, int ndst, const int *cell, double2 *out, cudaStream_t s)
{
    finalize<FIN_ADD>(partial, nsplit, ndst, cell, nullptr, nullptr, out, s);
}

void launch_finalize_f2f(const double2 *partial, int nsplit, int ndst, const int *cell, double2 *Pout, double2 *P,
                         cudaStream_t s)
{
    finalize<FIN_F2F>(partial, nsplit, ndst, cell, nullptr, Pout, P, s);
}

void launch_finalize_resp(const double2 *partial, int nsplit, int ndst, const int *cell, const double2 *gate_pin,
                          double2 *Pout, double2 *P, cudaStream_t s)
{
    finalize<FIN_RESP>(partial, nsplit, ndst, cell, gate_pin, Pout, P, s);
}

// Splits of a sum.  Scalar kernels: tiles over the splits, at least two to
// one.  Packed ones (the readout, target -> field object, target -> target):
// about 16 waves of resident CTAs, so that the uneven tiles (most
// blocks of a shadowed hop are empty) balance; with fewer tiles than that one
// tile to a split, and each tile's words over up to eight CTAs until there are
// two waves.
SumSplit sum_split(int hop, int rel, int ntiles, int ndstblocks, int nsm, int force)
{
    SumSplit s{1, 1, 1};
    const bool packed = !rel && (hop == HOP_FP || hop == HOP_NORESP || hop == HOP_RESP);
    const int nb = std::max(ndstblocks, 1), nt = std::max(ntiles, 1), slots = 3 * std::max(nsm, 1);
    int n = packed ? std::min(nt, (16 * slots + nb - 1) / nb) : std::max(1, std::min((2432 + nb - 1) / nb, nt / 2));
    if (force > 0) n = std::min(force, nt);
    s.tiles_per_split = (nt + n - 1) / n;
    const int tsplit = (nt + s.tiles_per_split - 1) / s.tiles_per_split;
    if (packed && force <= 0 && s.tiles_per_split == 1)
        while (s.wsplit < kWordsPerTile && (long long)nb * nt * s.wsplit < 2LL * slots) s.wsplit *= 2;
    s.nsplit = tsplit * s.wsplit;
    return s;
}

}  // namespace sonar
