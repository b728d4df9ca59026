// noalloc.cu -- fragment -> field-point readout that allocates no memory.
//
// Who needs it: callers that cannot call cudaMalloc while the readout runs.
// Typical cases are a host framework that owns every device byte through its
// own pool and forbids other allocations, a real-time or embedded host that
// allocates only at start-up, and code that must not trigger the implicit
// synchronisation a cudaMalloc/cudaFree can cause.  Such a caller keeps its
// own device buffers for the inputs and the outputs and calls
// sonar_readout_noalloc with them.
//
// What it computes: the FIELD_POINTS sum of ProjectTargetToFieldPoints
// (the reference's projectFacetToFieldPoints, src/OptiX.cu:112-190), for
// fragments and field points given as plain device arrays, without shadowing
// (every fragment sees every field point, subject to the area gate
// A > 1e-6 and the cos_scat >= 1e-6 gate, both decided with the reference's
// FP32 rounding as in the library's interaction masks).  For scenes where
// nothing occludes the readout -- flat or convex targets seen from outside --
// the result equals the library's own readout.
//
// Scratch: the only working memory is the per-split partial sums, held in a
// file-scope __device__ array of kMaxPartials double2 (8 MiB).  Every GPU that
// loads this library reserves that array until the process exits.  Its
// device address is looked up on the first call made in each CUDA context
// (cudaGetSymbolAddress, with that device current) and cached under the
// context's unique id: a context that is destroyed and re-created (for
// example by cudaDeviceReset) gets the array at a new address, which the
// next call looks up again.  Make the first call in a context before any
// stream capture begins.  Every call reuses the same array, which keeps the
// previous call's contents: the sum kernel overwrites every partial it later
// reads, so nothing needs clearing, but two calls whose work overlaps on the
// GPU (for example on two streams) race on the array and give wrong results.
#include <climits>
#include <cstdint>
#include <cstdio>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/sonar_render.h"
#include "pack2.cuh"

namespace sonar {
namespace {

constexpr int kMaxPartials = 1 << 19;  // double2 entries: 8 MiB
constexpr int kBlock = 256;
constexpr int kGroup = 2;              // source pairs whose gates share a vote
constexpr int kWord = 32;              // sources of a word, the unit of the splits
constexpr int kMaxDevices = 64;
constexpr int kMaxSplit = 1024;
constexpr int kSms = 152;              // SMs of the part this library is built for (sizes the grid only)

static __device__ __align__(256) double2 g_noalloc_partials[kMaxPartials];

// host-side cache of the array's device address, one entry per device: the
// address and the unique id of the context it was looked up in
struct PartialsAddr {
    unsigned long long ctx_id;
    double2 *ptr;
};
PartialsAddr g_partials_addr[kMaxDevices] = {};

constexpr float kInv4PiN = 0.0795774715459476679f;
constexpr float kTwoPiN = 6.28318530717958647692f;

__device__ __forceinline__ float dot3_rn(float ax, float ay, float az, float bx, float by, float bz)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(ax, bx), __fmul_rn(ay, by)), __fmul_rn(az, bz));
}

// cos_scat >= 1e-6 (src/OptiX.cu:155-160) decided as the reference rounds it:
// the contracted estimate est decides outside the band [0, 2e-6] (it is
// within a few ulp of the true cosine); inside the band the reference's
// expression is evaluated with every operation rounded separately --
// r = sqrt(v.v), u = v * (1 / r), dot(u, n).
__device__ __forceinline__ bool cos_scat_gate(float est, float vx, float vy, float vz, float nx, float ny, float nz)
{
    if (est > 2e-6f) return true;
    if (est < 0.0f) return false;
    const float r = __fsqrt_rn(dot3_rn(vx, vy, vz, vx, vy, vz));
    const float inv = __frcp_rn(r);
    return !(dot3_rn(__fmul_rn(vx, inv), __fmul_rn(vy, inv), __fmul_rn(vz, inv), nx, ny, nz) < 1e-6f);
}

struct Wave {
    float kr, ka, k2hi, k2lo;
};

// One pair by the scalar expressions: its gate and term added to fr, fi.
__device__ __forceinline__ void scalar_pair(const Wave &k, float px, float py, float pz, float4 A, float4 B, float &fr,
                                            float &fi)
{
    const float vx = __fsub_rn(px, A.x), vy = __fsub_rn(py, A.y), vz = __fsub_rn(pz, A.z);
    const float r2 = dot3_rn(vx, vy, vz, vx, vy, vz);
    const float r = __fsqrt_rn(r2);
    const float rinv = rsqrtf(r2);
    const float cs = (vx * B.x + vy * B.y + vz * B.z) * rinv;  // cos_scat, src/OptiX.cu:155
    if ((A.w == 0.0f && B.w == 0.0f) || !cos_scat_gate(cs, vx, vy, vz, B.x, B.y, B.z)) return;
    const float th = __fmul_rn(r, k.k2hi);
    const float tl = fmaf(r, k.k2lo, fmaf(r, k.k2hi, -th));
    const float frac = (th - rintf(th)) + tl;
    float sn, cn;
    __sincosf(frac * kTwoPiN, &sn, &cn);
    float amp = rinv * kInv4PiN;
    if (k.ka != 0.0f) amp *= __expf(-k.ka * r);
    // -e^{ikr}/(4 pi) (ik/r) + 1/r^2  (src/OptiX.cu:182)
    const float gr = fmaf(amp, fmaf(k.ka, cn, k.kr * sn), rinv * rinv) * cs;
    const float gi = amp * fmaf(k.ka, sn, -k.kr * cn) * cs;
    fr += gr * A.w - gi * B.w;
    fi += gr * B.w + gi * A.w;
}

// Staged source pairs [q0, q1) one by one (s: four arrays of kBlock / 2).
__device__ __noinline__ float2 scalar_pairs(const Wave &k, const float4 *s, int q0, int q1, float px, float py, float pz)
{
    float fr = 0.0f, fi = 0.0f;
#pragma unroll 1
    for (int q = q0; q < q1; ++q) {
        const float4 a = s[q], b = s[kBlock / 2 + q], c = s[kBlock + q], d = s[3 * kBlock / 2 + q];
        scalar_pair(k, px, py, pz, make_float4(a.x, a.z, b.x, b.z), make_float4(d.x, d.z, c.z, c.x), fr, fi);
        scalar_pair(k, px, py, pz, make_float4(a.y, a.w, b.y, b.w), make_float4(d.y, d.w, c.w, c.y), fr, fi);
    }
    return make_float2(fr, fi);
}

// One CTA: 256 field points x the source words [w0, w1) of its split.  Same
// arithmetic as the library's packed readout sum (two sources to a register);
// the area and cos_scat gates are evaluated inline instead of being read from
// an interaction mask.  A pair whose estimate leaves its gate open, whose
// distance FP32 cannot square, and every pair of a tile with a weight that is
// not finite (or of a wave number the packed form cannot divide by, or whose
// packed sum leaves FP32) takes scalar_pair.  An estimate below 2.5e-7 fails
// for certain (it is within 7e-7 of the exact cosine), so fragments without
// area, staged with a zero normal, never reach the open band.  The distance,
// one Newton step on the approximate reciprocal root, equals the correctly
// rounded square root: compared on the part for all 1.91e9 FP32 arguments from
// 1e-30 up.  A chunk's sum is FP32, what adds up the chunks FP64.
//
// What bounds it: FP32 lanes (70 % of the pipe's cycles, 33 operations a pair)
// beside 3 special-function operations (4 with attenuation, 61 % of that
// unit); the scalar form was bound by issue, about 85 instructions (IEEE
// square root, a branch per gate).  62,003 fragments x 40,001 points with
// attenuation: 5.69 -> 3.41 ms; 1,271 x 181 from 5 CTAs to 40: 47 -> 7 us.
// Measured and left out, with the scalar pairs in the loop (3.45 ms): groups of 1
// (3.52) and 4 (4.06).
template <bool ATT>
__global__ void __launch_bounds__(kBlock, 3)
    k_readout_noalloc(const float4 *__restrict__ pos, const float4 *__restrict__ nrm,
                      const double2 *__restrict__ pres, int nsrc, const float4 *__restrict__ pts, int ndst, Wave k,
                      int packed_ok, int nwords, int words_per_split, double2 *partials)
{
    // pairs of sources: (x0 x1 y0 y1) (z0 z1 wr0 wr1) (wi0 wi1 nz0 nz1) (nx0 nx1 ny0 ny1)
    __shared__ float4 sS[4][kBlock / 2];
    const int tid = threadIdx.x;
    const int j = blockIdx.x * kBlock + tid;
    const bool live = j < ndst;
    const float4 p = pts[live ? j : blockIdx.x * kBlock];
    const f2 px = dup2(p.x), py = dup2(p.y), pz = dup2(p.z);
    const float kr4pi = k.kr * kInv4PiN;
    const Phase2 ph = phase2(k.k2hi, k.k2lo);
    const f2 half = dup2(0.5f), c4pik = dup2(1.0f / kr4pi);
    const f2 natt = dup2(-k.ka * 1.44269504088896341f), qatt = dup2(k.ka / k.kr), nqatt = dup2(-(k.ka / k.kr));
    double accr = 0.0, acci = 0.0;
    const int w0 = blockIdx.y * words_per_split, w1 = min(w0 + words_per_split, nwords);
    for (int wb = w0; wb < w1; wb += kBlock / kWord) {
        const int i0 = wb * kWord;
        int npair = (min(min(w1 - wb, kBlock / kWord) * kWord, nsrc - i0) + 1) / 2;
        npair = (npair + kGroup - 1) / kGroup * kGroup;  // at most the 128 the arrays hold
        __syncthreads();
        bool fin = true;
        if (tid < npair) {
            float4 A[2], B[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int i = i0 + 2 * tid + s;
                const float4 q = pos[i < nsrc ? i : i0];
                // fragments below the area gate (src/OptiX.cu:138) and past the end: no weight, zero normal
                A[s] = make_float4(q.x, q.y, q.z, 0.0f);
                B[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (i < nsrc && q.w > 1e-6f) {
                    const float4 n = nrm[i];
                    const double2 w = pres[i];
                    A[s].w = (float)((double)q.w * w.x);
                    B[s] = make_float4(n.x, n.y, n.z, (float)((double)q.w * w.y));
                    if (A[s].w == 0.0f && B[s].w == 0.0f) B[s] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    fin = fin && fabsf(A[s].w) <= 3.0e38f && fabsf(B[s].w) <= 3.0e38f;
                }
            }
            sS[0][tid] = make_float4(A[0].x, A[1].x, A[0].y, A[1].y);
            sS[1][tid] = make_float4(A[0].z, A[1].z, A[0].w, A[1].w);
            sS[2][tid] = make_float4(B[0].w, B[1].w, B[0].z, B[1].z);
            sS[3][tid] = make_float4(B[0].x, B[1].x, B[0].y, B[1].y);
        }
        const bool packed = __syncthreads_and(fin) && packed_ok;
        f2 acc[3] = {0ull, 0ull, 0ull};
        float fr = 0.0f, fi = 0.0f;
        // kGroup source pairs at a time: their gates under one vote, so that the
        // distances of a group and the phases of the one before overlap
#pragma unroll 2
        for (int q0 = 0; q0 < npair; q0 += kGroup) {
            f2 r2[kGroup], rinv[kGroup], d1[kGroup];
            bool on[2 * kGroup], slow = !packed;
#pragma unroll
            for (int u = 0; u < kGroup; ++u) {
                const int q = q0 + u;  // past npair: staged without weight
                const ulonglong2 XY = *reinterpret_cast<const ulonglong2 *>(&sS[0][q]);
                const f2 Z = *reinterpret_cast<const f2 *>(&sS[1][q]);
                const f2 NZ = *(reinterpret_cast<const f2 *>(&sS[2][q]) + 1);
                const ulonglong2 NN = *reinterpret_cast<const ulonglong2 *>(&sS[3][q]);
                const f2 vx = sub2(px, XY.x), vy = sub2(py, XY.y), vz = sub2(pz, Z);
                r2[u] = dot_rn2(vx, vy, vz);
                rinv[u] = rsqrt2(r2[u]);
                d1[u] = fma2(vx, NN.x, fma2(vy, NN.y, mul2(vz, NZ)));
                float c0, c1, x0, x1;
                up2(mul2(d1[u], rinv[u]), c0, c1);
                up2(r2[u], x0, x1);
                on[2 * u] = c0 > 2e-6f;
                on[2 * u + 1] = c1 > 2e-6f;
                slow = slow || (!on[2 * u] && !(c0 < 2.5e-7f)) || (!on[2 * u + 1] && !(c1 < 2.5e-7f)) ||
                       !(fminf(x0, x1) > 1e-30f);
            }
            if (__any_sync(0xffffffffu, slow)) {
                const float2 v = scalar_pairs(k, &sS[0][0], q0, q0 + kGroup, p.x, p.y, p.z);
                fr += v.x;
                fi += v.y;
                continue;
            }
#pragma unroll
            for (int u = 0; u < kGroup; ++u) {
                const f2 WR = *(reinterpret_cast<const f2 *>(&sS[1][q0 + u]) + 1);
                const f2 WI = *reinterpret_cast<const f2 *>(&sS[2][q0 + u]);
                const f2 r0 = mul2(r2[u], rinv[u]);
                const f2 r = fma2(fma2(r0 ^ 0x8000000080000000ull, r0, r2[u]), mul2(rinv[u], half), r0);
                f2 f = fma2(r, ph.khi, sub2(ph.magic, fma2(r, ph.khi, ph.magic)));
                f = mul2(fma2(r, ph.klo, f), ph.two_pi);
                float f0, f1, s0, s1, e0, e1;
                up2(f, f0, f1);
                __sincosf(f0, &s0, &e0);
                __sincosf(f1, &s1, &e1);
                const f2 sn = pk2(s0, s1), cs = pk2(e0, e1);
                const f2 amp = mul2(mul2(rinv[u], rinv[u]), d1[u]);  // (4 pi / k) cos_scat / r
                f2 Tr, Ti;
                if (ATT) {
                    const f2 osc = mul2(amp, ex2_2(mul2(r, natt)));
                    Tr = fma2(osc, fma2(qatt, cs, sn), mul2(amp, mul2(rinv[u], c4pik)));
                    Ti = mul2(osc, fma2(nqatt, sn, cs));
                } else {
                    Tr = mul2(amp, fma2(rinv[u], c4pik, sn));
                    Ti = mul2(amp, cs);
                }
                float a0, a1, b0, b1;
                up2(Tr, a0, a1);
                up2(Ti, b0, b1);
                Tr = pk2(on[2 * u] ? a0 : 0.0f, on[2 * u + 1] ? a1 : 0.0f);
                Ti = pk2(on[2 * u] ? b0 : 0.0f, on[2 * u + 1] ? b1 : 0.0f);
                acc[0] = fma2(Tr, WR, fma2(Ti, WI, acc[0]));
                acc[1] = fma2(Tr, WI, acc[1]);
                acc[2] = fma2(Ti, WR, acc[2]);
            }
        }
        if (packed) {
            fr = fmaf(kr4pi, sum2(acc[0]), fr);
            fi = fmaf(kr4pi, sum2(acc[1]) - sum2(acc[2]), fi);
            if (!(fabsf(fr) <= 3.0e38f && fabsf(fi) <= 3.0e38f)) {
                // k / (4 pi) is left to the end of the packed sum, which can
                // leave FP32 where the sum itself does not
                const float2 v = scalar_pairs(k, &sS[0][0], 0, npair, p.x, p.y, p.z);
                fr = v.x;
                fi = v.y;
            }
        }
        accr += (double)fr;
        acci += (double)fi;
    }
    if (live) partials[(long long)blockIdx.y * ndst + j] = make_double2(accr, acci);
}

// out += the splits' partials, in SHARES contiguous shares added in order (a
// thread that reads many splits one after the other is bound by that chain).
template <int SHARES>
__global__ void __launch_bounds__(kBlock) k_readout_noalloc_finalize(const double2 *partials, int nsplit, int ndst,
                                                                    double2 *out)
{
    constexpr int kDst = kBlock / SHARES;
    __shared__ double2 sS[SHARES][kDst];
    const int l = threadIdx.x % kDst, g = threadIdx.x / kDst;
    const int j = blockIdx.x * kDst + l;
    double sr = 0.0, si = 0.0;
    if (j < ndst)
        for (int k = nsplit * g / SHARES; k < nsplit * (g + 1) / SHARES; ++k) {
            const double2 v = partials[(long long)k * ndst + j];
            sr += v.x;
            si += v.y;
        }
    if (SHARES > 1) {
        sS[g][l] = make_double2(sr, si);
        __syncthreads();
    }
    if (g > 0 || j >= ndst) return;
#pragma unroll 8
    for (int k = 1; k < SHARES; ++k) {
        sr += sS[k][l].x;
        si += sS[k][l].y;
    }
    double2 o = out[j];
    o.x += sr;
    o.y += si;
    out[j] = o;
}

// Splits of the source words: among the counts the scratch and the words
// allow, up to 16 waves of resident CTAs (three to an SM), the largest of
// those whose last wave is fullest.
int choose_splits(int nblocks, int nwords, int n_points, int nsm)
{
    const int slots = 3 * nsm;
    long long most = kMaxPartials / n_points;
    most = most > kMaxSplit ? kMaxSplit : most;
    most = most > nwords ? nwords : most;
    const long long waves = (16LL * slots + nblocks - 1) / nblocks;
    most = most > waves ? waves : most;
    int best = 1;
    double eff = 0.0;
    for (int n = 1; n <= (int)most; ++n) {
        const double x = (double)nblocks * n / slots, e = x / (double)((long long)(x + 0.999999));
        // fewer CTAs than slots: the more the better
        if (x <= 1.0 || e >= eff - 0.01) {
            best = n;
            eff = x <= 1.0 ? e : (e > eff ? e : eff);
        }
    }
    return best;
}

// Unique id of the calling thread's current CUDA context (0 when none is
// current), through the driver entry points the runtime hands out (the
// library does not link the driver library itself).
unsigned long long current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    if (!get_current || !get_id) {
        void *f0 = nullptr, *f1 = nullptr;
        cudaDriverEntryPointQueryResult q0, q1;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f0, 12000, cudaEnableDefault, &q0) != cudaSuccess ||
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f1, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
            q0 != cudaDriverEntryPointSuccess || q1 != cudaDriverEntryPointSuccess || !f0 || !f1)
            return 0;
        get_current = (GetCurrent)f0;
        get_id = (GetId)f1;
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx) return 0;
    if (get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// Device address of the partials array in the current context, looked up
// on the first call made in that context.
int partials_for_current_device(double2 **out)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SONAR_NOALLOC_ECUDA;
    unsigned long long id = current_context_id();
    PartialsAddr &c = g_partials_addr[dev];
    if (id == 0 || c.ctx_id != id || !c.ptr) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);  // makes the context current
        if (e != cudaSuccess || !p) {
            fprintf(stderr, "sonar_readout_noalloc: cudaGetSymbolAddress failed: %s\n", cudaGetErrorString(e));
            return SONAR_NOALLOC_ECUDA;
        }
        id = current_context_id();
        c.ctx_id = id;  // 0 (no id available): looked up again on every call
        c.ptr = (double2 *)p;
    }
    *out = c.ptr;
    return 0;
}

bool misaligned16(const void *p) { return ((uintptr_t)p & 15u) != 0; }

}  // namespace
}  // namespace sonar

using namespace sonar;

extern "C" int sonar_readout_noalloc(const float *frag_pos, const float *frag_normal, const double *frag_pressure,
                                     int n_frag, const float *points, int n_points, float k_re, float k_im,
                                     double *out, void *stream)
{
    if (n_frag < 0 || n_points < 0 || n_frag > INT_MAX - kBlock) return SONAR_NOALLOC_EINVAL;
    if (n_points > SONAR_NOALLOC_MAX_POINTS) {
        fprintf(stderr, "sonar_readout_noalloc: %d field points exceed the maximum of %d\n", n_points,
                SONAR_NOALLOC_MAX_POINTS);
        return SONAR_NOALLOC_ETOOBIG;
    }
    if (n_points == 0) return 0;
    if (!points || !out || (n_frag > 0 && (!frag_pos || !frag_normal || !frag_pressure))) return SONAR_NOALLOC_EINVAL;
    // the kernels read float4 / double2 vectors: every buffer 16-byte aligned
    if (misaligned16(points) || misaligned16(out) ||
        (n_frag > 0 && (misaligned16(frag_pos) || misaligned16(frag_normal) || misaligned16(frag_pressure)))) {
        fprintf(stderr, "sonar_readout_noalloc: every buffer must start on a 16-byte boundary\n");
        return SONAR_NOALLOC_EINVAL;
    }
    // an error left pending by the caller's own work is reported, not taken over
    const cudaError_t prior = cudaPeekAtLastError();
    if (prior != cudaSuccess) {
        fprintf(stderr, "sonar_readout_noalloc: a CUDA error is already pending: %s\n", cudaGetErrorString(prior));
        return SONAR_NOALLOC_ECUDA;
    }
    double2 *partials = nullptr;
    const int st = partials_for_current_device(&partials);
    if (st != 0) return st;
    if (n_frag == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const int nwords = (n_frag + kWord - 1) / kWord;
    const int nblocks = (n_points + kBlock - 1) / kBlock;
    int nsplit = choose_splits(nblocks, nwords, n_points, kSms);
    const int wps = (nwords + nsplit - 1) / nsplit;
    nsplit = (nwords + wps - 1) / wps;
    const double k2 = (double)k_re / (2.0 * 3.14159265358979323846);
    const float k2hi = (float)k2, k2lo = (float)(k2 - (double)k2hi);
    const Wave k{k_re, k_im, k2hi, k2lo};
    // the packed form divides by k
    const int packed_ok = k_re > 1e-11f && k_re < 1e11f && k_im >= 0.0f && k_im <= 1e6f * k_re;
    const dim3 grid(nblocks, nsplit);
    const float4 *fp = (const float4 *)frag_pos, *fn = (const float4 *)frag_normal, *pt = (const float4 *)points;
    const double2 *pr = (const double2 *)frag_pressure;
    if (k_im != 0.0f)
        k_readout_noalloc<true><<<grid, kBlock, 0, s>>>(fp, fn, pr, n_frag, pt, n_points, k, packed_ok, nwords, wps,
                                                       partials);
    else
        k_readout_noalloc<false><<<grid, kBlock, 0, s>>>(fp, fn, pr, n_frag, pt, n_points, k, packed_ok, nwords, wps,
                                                        partials);
    if (nsplit >= 128)
        k_readout_noalloc_finalize<32><<<(n_points + 7) / 8, kBlock, 0, s>>>(partials, nsplit, n_points, (double2 *)out);
    else if (nsplit >= 16)
        k_readout_noalloc_finalize<8><<<(n_points + 31) / 32, kBlock, 0, s>>>(partials, nsplit, n_points, (double2 *)out);
    else
        k_readout_noalloc_finalize<1><<<nblocks, kBlock, 0, s>>>(partials, nsplit, n_points, (double2 *)out);
    const cudaError_t e = cudaPeekAtLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "sonar_readout_noalloc: launch failed: %s\n", cudaGetErrorString(e));
        return SONAR_NOALLOC_ECUDA;
    }
    return 0;
}
