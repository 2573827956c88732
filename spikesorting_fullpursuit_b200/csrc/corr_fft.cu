// corr_fft.cu -- template correlations by 256-point transforms (fft256.cuh): the
// template-by-voltage likelihood and the partial correlations of the overlap
// recheck.
//
// A template spans W samples on a few channels; correlating it with the voltage
// directly takes W multiply-adds per sample, channel and template.  By transforms a
// stretch's channels are transformed once, and each template costs one product per
// frequency and channel and one inverse transform.
#include <algorithm>

#include "fft256.cuh"
#include "lik_common.cuh"

namespace fbp {
namespace {

constexpr size_t kFftSmemMost = 222 * 1024;   // dynamic shared memory of a CTA
constexpr size_t kSpecMost = 2ull << 30;      // bytes of template spectra

// Per template, one warp: its non-zero channels, their norms (rounded up; 0 for an
// all-zero channel), the channel mask (all ones above 64 channels), the taps padded to a multiple of 4 (exact
// recomputation), and the bound of the likelihood's estimate,
//     lbnd.x sum_c |T_c| |z_c| + lbnd.y |bias|
// (the reference's sequential sum of n W products, then the transforms, over the
// n non-zero channels).
__global__ void template_info_kernel(Dims d, const float* __restrict__ T, uint8_t* clist, uint32_t* ccnt,
                                     float* tnorm, unsigned long long* tchm, float* Tp, float2* lbnd)
{
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5, Wp = (d.W + 3) & ~3u;
    const float u = 1.0f / 16777216.0f;
    for (uint32_t t = blockIdx.x * wpb + (threadIdx.x >> 5); t < d.M; t += gridDim.x * wpb) {
        uint32_t n = 0;
        unsigned long long mask = 0ull;
        for (uint32_t c = 0; c < d.C; ++c) {
            const uint64_t tc = (uint64_t)t * d.C + c;
            const float* r = T + tc * d.W;
            bool nz = false;
            double a = 0.0;
            for (uint32_t j = lane; j < Wp; j += 32) {
                const float v = j < d.W ? r[j] : 0.f;
                Tp[tc * Wp + j] = v;
                nz |= v != 0.f;
                a += (double)v * v;
            }
            nz = __any_sync(0xffffffffu, nz);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
            if (lane == 0) {
                tnorm[tc] = (float)(sqrt(a) * (1.0 + 1e-6));
                if (nz) clist[(size_t)t * d.C + n] = (uint8_t)c;
            }
            if (nz) {
                ++n;
                if (c < 64) mask |= 1ull << c;
            }
        }
        if (lane == 0) {
            ccnt[t] = n;
            tchm[t] = d.C <= 64 ? mask : ~0ull;   // more than 64 channels: nothing is skipped by it
            lbnd[t] = make_float2(1.05f * u * ((float)n * d.W + 6.f + kFftTerms + 3.f * n), 1.05f * u * ((float)n * d.W + 8.f));
        }
    }
}

// Spectra (after template_info_kernel) and the twiddle table, one CTA per (template,
// place in its channel list).
__global__ void __launch_bounds__(kFft) spectra_kernel(Dims d, const float* __restrict__ T,
                                                       const uint8_t* __restrict__ clist,
                                                       const uint32_t* __restrict__ ccnt, float4* spec, float2* tw)
{
    __shared__ double2 w[kFft];   // e^(-2 pi i k / 256)
    __shared__ float x[128];
    const uint32_t t = blockIdx.x / d.C, i = blockIdx.x % d.C, k = threadIdx.x;
    const bool any = i < ccnt[t];
    if (!any && blockIdx.x != 0) return;
    double sn, cs;
    sincospi(-2.0 * k / kFft, &sn, &cs);
    w[k] = make_double2(cs, sn);
    if (blockIdx.x == 0) {   // twiddles e^(2 pi i l r / 256) at r * 16 + l
        sincospi(2.0 * ((k & 15u) * (k >> 4)) / kFft, &sn, &cs);
        tw[k] = make_float2((float)cs, (float)sn);
    }
    if (any && k < d.W) x[k] = T[((uint64_t)t * d.C + clist[blockIdx.x]) * d.W + k];
    __syncthreads();
    if (!any) return;
    double re = 0.0, im = 0.0;
    for (uint32_t j = 0; j < d.W; ++j) {
        const double2 e = w[(j * k) & (kFft - 1)];
        re = fma((double)x[j], e.x, re);
        im = fma((double)x[j], e.y, im);
    }
    // k = l + 32 m (+ 16): element (m, l), first or second half of the float4
    float2* o = reinterpret_cast<float2*>(spec + (size_t)blockIdx.x * 128 + (k >> 5) * 16 + (k & 15u));
    o[(k >> 4) & 1u] = make_float2((float)(re / kFft), (float)(im / kFft));
}

// A window's energy e on a channel is not a finite number: its samples are zeroed
// (PART 0 the real, 1 the imaginary parts), and the energy becomes NaN if a sample is
// not finite, infinite if only the squares overflow.  By whole half-warps.
template <int PART>
__device__ __forceinline__ float keep_apart(float2 (&x)[16], float e)
{
    if (e < INFINITY) return e;
    bool wild = false;
#pragma unroll
    for (int m = 0; m < 16; ++m) {
        float& v = PART ? x[m].y : x[m].x;
        wild |= !(fabsf(v) < INFINITY);
        v = 0.f;
    }
    return __any_sync(0xFFFFu << (threadIdx.x & 16u), wild) ? __int_as_float(0x7fffffff) : INFINITY;
}

// Partial correlations of flagged windows (see overlap_fast.cu):
//     G[k][t][b] = X_t(b) - 0.5 Et[t][b],   X_t(b) = sum_cj T[t][c][j - (b - S)] v[c][j]
// over the window's W samples, the window's energy per channel, vc2[k][c], and that of
// the signals transformed together, z2[k][c].  A CTA takes two windows at a time (kk = 2 u, 2 u + 1 of the batch) as one complex signal:
// the windows, zero-padded to 256, are transformed channel by channel, then each
// half-warp correlates its templates.  A window needs W + min(S, W - 1) <= 256: a
// shift's samples then never wrap onto another's.
//
// Bounded by latency (ncu, 16 channels x 40 templates: 42 % of the issue slots, L1
// 54 %, L2 20 %, DRAM 9 % of their peaks, 24 warps per SM): the spectra stream from
// L2 into registers, each value used for two windows.
template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) window_corr_kernel(
    Dims d, FftTables F, const float* __restrict__ V, const float* __restrict__ L, const float* __restrict__ theta,
    const float2* __restrict__ Et, const uint32_t* __restrict__ flag, DevStatus* status,
    const uint32_t* __restrict__ best_lab, const uint32_t* __restrict__ best_idx, uint32_t k0, uint32_t kc, float* G,
    float* vc2, float* z2)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const uint32_t nh = blockDim.x >> 4;
    float4* zs = reinterpret_cast<float4*>(smraw);                     // [C][8][16]
    float2* xbuf = reinterpret_cast<float2*>(zs + (size_t)d.C * 128);  // [nh][256]
    float2* tw = xbuf + (size_t)nh * kFft;                             // [256]
    const uint32_t l = threadIdx.x & 15u, h = threadIdx.x >> 4;
    const uint32_t S = d.S, W = d.W, M = d.M, S2 = 2 * S + 1;
    const uint32_t Sw = S < W - 1 ? S : W - 1;   // shifts beyond meet no sample
    for (uint32_t i = threadIdx.x; i < kFft; i += blockDim.x) tw[i] = F.tw[i];
    const uint32_t nflag = flagged_windows(status);
    const uint32_t live = nflag > k0 ? min(kc, nflag - k0) : 0u;
    unsigned long long macs = 0;
    for (uint32_t u = blockIdx.x; 2 * u < live; u += gridDim.x) {
        uint32_t p[2];
        bool ok[2];
#pragma unroll
        for (uint32_t w = 0; w < 2; ++w) {
            const uint32_t kk = 2 * u + w;
            ok[w] = false;
            p[w] = 0;
            if (kk < live) {
                const uint32_t id = flag[k0 + kk], f = best_lab[id];
                p[w] = best_idx[id];
                ok[w] = !(L[(uint64_t)f * d.N + p[w]] < theta[f] || (uint64_t)p[w] >= (uint64_t)d.N - W);
            }
        }
        if (!ok[0] && !ok[1]) continue;
        __syncthreads();   // the spectra of the previous pair are read
        float2 x[16];
        for (uint32_t c0 = 0; c0 < d.C; c0 += nh) {
            const uint32_t c = c0 + h;
            if (c0 + (h & ~1u) >= d.C) continue;   // the whole warp
            const bool on = c < d.C;
            const float* vr = V + (uint64_t)(on ? c : 0u) * d.N;
            float ea = 0.f, eb = 0.f;
#pragma unroll
            for (uint32_t m = 0; m < 16; ++m) {
                const uint32_t j = l + 16 * m;
                x[m].x = (on && ok[0] && j < W) ? vr[p[0] + j] : 0.f;
                x[m].y = (on && ok[1] && j < W) ? vr[p[1] + j] : 0.f;
                ea = fmaf(x[m].x, x[m].x, ea);
                eb = fmaf(x[m].y, x[m].y, eb);
            }
            ea = half_sum(ea);
            eb = half_sum(eb);
            if (!(ea + eb < INFINITY)) {   // keep what is not finite, or overflows, off the other window
                ea = keep_apart<0>(x, ea);
                eb = keep_apart<1>(x, eb);
            }
            __syncwarp();
            if (on && l == 0) {
                const size_t at = (size_t)(2 * u) * d.C + c;
                const float z = (ea < INFINITY ? ea : 0.f) + (eb < INFINITY ? eb : 0.f);
                if (2 * u < live) { vc2[at] = ea; z2[at] = z; }
                if (2 * u + 1 < live) { vc2[at + d.C] = eb; z2[at + d.C] = z; }
            }
            // an idle half-warp of the last channels exchanges through a spare buffer
            fft_channel(x, on ? zs + (size_t)c * 128 : reinterpret_cast<float4*>(xbuf + (size_t)h * kFft), tw, l);
        }
        FftAhead A;
        fft_fetch(F, d.C, h < M ? h : 0u, h < M, l, A);
        __syncthreads();
        float* Ga = G + (uint64_t)(2 * u) * M * S2;
        float* Gb = Ga + (uint64_t)M * S2;
        for (uint32_t t0 = 0; t0 + (h & ~1u) < M; t0 += nh) {
            const uint32_t t = t0 + h;
            const bool on = t < M;
            if (l == 0) macs += 4ull * kFft * A.cnt;
            fft_correlate(F, d.C, on ? t : 0u, A, t + nh, t + nh < M, zs, xbuf + (size_t)h * kFft, tw, l, x);
            if (!on) continue;
            const float2* et = Et + (uint64_t)t * S2;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) {
                const uint32_t y = (16 * q + l + Sw) & (kFft - 1);   // output n is shift n, or n - 256
                if (y > 2 * Sw) continue;
                const uint32_t b = y + S - Sw;
                const float e = 0.5f * et[b].x;
                if (ok[0]) Ga[(uint64_t)t * S2 + b] = x[q].x - e;
                if (ok[1]) Gb[(uint64_t)t * S2 + b] = x[q].y - e;
            }
            for (uint32_t y = l; y < 2 * (S - Sw); y += 16) {   // no overlap with the window
                const uint32_t b = y < S - Sw ? y : S2 - 1 - (y - (S - Sw));
                if (ok[0]) Ga[(uint64_t)t * S2 + b] = 0.f;
                if (ok[1]) Gb[(uint64_t)t * S2 + b] = 0.f;
            }
        }
    }
    if (macs) atomicAdd(&status->pc_macs, macs);
}

// ---------------------------------------------------------------------------
// Likelihood.  L[t][s] = bias[t] + sum_c sum_j T[t][c][j] V[c][s + j]
// (compute_full_likelihood, binary_pursuit.cl:216-300) by overlap-save: a stretch of
// 256 samples gives Vn = 257 - W likelihood samples of every template.  A CTA takes
// spans of two stretches (2 Vn samples) as one complex signal: for the whole chunk
// consecutive spans, else spans cut from the runs of listed windows (units).
//
// Lazy exactness (the pursuit), as in lik_tc.cu: an estimate is off the reference's
// float value by at most bnd (lbnd, fft256.cuh; about 4e-5 of sum |T_c| |z_c|,
// z the pair of stretches).  Samples of uncertain sign are queued for the exact
// recomputation (fixup kernel); samples certainly <= 0 keep their estimate; of the
// certainly positive ones, those whose upper bound reaches the largest lower bound of
// their window (within the stretch) are queued, the others keep their estimate and
// flag their (window, template) row.
//
// Measured per pursuit against the tensor-core kernel (TF32, 128-sample tiles), both
// with their exact recomputation: 16 channels x 40 templates, 300 s 32.5 -> 16.5 ms;
// 64 x 200, 20 s 81.2 -> 20.6 ms; 23 x 77, 41 s 17.2 -> 8.7 ms; without a zero channel
// 16 x 40 4.6 -> 3.2 ms, 64 x 200 43 -> 33 ms.  Bounded by the shared-memory and L1
// data pipe (63 % busy, 56 % of the issue slots, 23 warps per SM): the spectra of
// templates and signals are read for every product.
// ---------------------------------------------------------------------------
struct LikFft {
    Dims d;
    FftTables F;
    const float* V;
    const float* T;
    const float* bias;
    const float* tnorm;
    const float2* lbnd;
    const uint2* units;     // {first sample, samples <= 2 Vn}, or null: the whole chunk's spans
    uint32_t n_spans;       // spans (units == null)
    uint64_t span0;         // first span
    float* L;
    unsigned long long* fix;
    uint32_t fix_cap;
    DevStatus* status;
    unsigned long long* wkey;
    uint8_t* wpos;
    uint8_t* wflag;
    uint32_t wslots;        // windows a stretch's samples can touch
};

__host__ __device__ inline uint32_t lik_stretch(uint32_t W) { return kFft + 1 - W; }
__host__ __device__ inline uint32_t lik_slots(uint32_t W) { return (lik_stretch(W) + W - 1) / W + 1; }

// Queues the samples with `need` as runs of 4: lanes 4 g .. 4 g + 3 hold consecutive
// samples of one template.  Where the queue is full they are computed right here.
__device__ __noinline__ void queue_samples(const LikFft& P, bool need, uint32_t t, uint32_t s)
{
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31;
    const uint32_t m = __ballot_sync(full, need);
    if (m == 0u) return;
    const uint32_t nib = (m >> (lane & ~3u)) & 0xFu;
    const bool lead = nib != 0u && (lane & 3u) == 0u;
    const uint32_t lm = __ballot_sync(full, lead);
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(&P.status->n_fix, __popc(lm));
    uint32_t at = __shfl_sync(full, base, 0) + __popc(lm & ((1u << lane) - 1u));
    if (lead && at < P.fix_cap) P.fix[at] = ((unsigned long long)t << 40) | ((unsigned long long)nib << 32) | s;
    at = __shfl_sync(full, at, lane & ~3u);
    if (need && at >= P.fix_cap) {
        const float v = exact_likelihood(P.d, P.V, P.T, P.bias[t], t, s, P.tnorm);
        P.L[(uint64_t)t * P.d.N + s] = v;
        note_window(P.d, P.wkey, P.wpos, v, t, s);
    }
}

// A certainly positive sample (t, s) with estimate v: queued if it can be its window's
// maximum (it reaches the window's largest lower bound mlb), else its row is flagged.
// Any lanes of a warp.
__device__ __forceinline__ void settle_positive(const LikFft& P, uint32_t t, uint32_t s, float v, float bd, float mlb)
{
    if (!(v + bd >= mlb)) {
        P.wflag[(uint64_t)(s / P.d.W) * P.d.M + t] = 1;
        return;
    }
    const uint32_t at = atomicAdd(&P.status->n_fix, 1u);
    if (at < P.fix_cap) {
        P.fix[at] = ((unsigned long long)t << 40) | (1ull << 32) | s;
        return;
    }
    const float e = exact_likelihood(P.d, P.V, P.T, P.bias[t], t, s, P.tnorm);
    P.L[(uint64_t)t * P.d.N + s] = e;
    note_window(P.d, P.wkey, P.wpos, e, t, s);
}

constexpr uint32_t kPosCap = 512;   // a span's certainly positive samples kept for the second look

template <int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) lik_fft_kernel(const __grid_constant__ LikFft P)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const Dims& d = P.d;
    const uint32_t nh = blockDim.x >> 4, C = d.C, M = d.M, W = d.W, Vn = lik_stretch(W), mw = (M + 31) / 32;
    float4* zs = reinterpret_cast<float4*>(smraw);                   // [C][8][16]
    float2* xbuf = reinterpret_cast<float2*>(zs + (size_t)C * 128);  // [nh][256]
    float2* tw = xbuf + (size_t)nh * kFft;                           // [256]
    float4* tpar = reinterpret_cast<float4*>(tw + kFft);             // [M] bias, lbnd.x, lbnd.y |bias|, the span's bound
    uint2* plist = reinterpret_cast<uint2*>(tpar + M);               // [kPosCap] {t << 9 | second << 8 | sample, estimate}
    float* nz = reinterpret_cast<float*>(plist + kPosCap);           // [C] norms of the pair of stretches
    int* s_mlb = reinterpret_cast<int*>(nz + C);                     // [2][wslots] largest lower bound (float bits)
    uint32_t* s_full = reinterpret_cast<uint32_t*>(s_mlb + 2 * P.wslots);   // [2][mw] templates with positives not in plist
    uint32_t* s_np = s_full + 2 * mw;
    const uint32_t l = threadIdx.x & 15u, h = threadIdx.x >> 4, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kFft; i += blockDim.x) tw[i] = P.F.tw[i];
    for (uint32_t t = threadIdx.x; t < M; t += blockDim.x) {
        const float b = P.bias[t];
        const float2 lb = P.lbnd[t];
        tpar[t] = make_float4(b, lb.x * 1.0001f, lb.y * fabsf(b), 0.f);
    }
    const uint32_t n = P.units ? P.status->n_units : P.n_spans;
    for (uint32_t k = blockIdx.x; k < n; k += gridDim.x) {
        uint32_t s0, total;
        if (P.units) {
            const uint2 un = P.units[k];
            s0 = un.x;
            total = un.y;
        } else {
            const uint64_t a = (P.span0 + k) * 2 * Vn;
            s0 = (uint32_t)a;
            total = (uint32_t)min((uint64_t)2 * Vn, (uint64_t)d.N - a);
        }
        __syncthreads();   // the previous span's shared state is read
        for (uint32_t i = threadIdx.x; i < 2 * P.wslots; i += blockDim.x) s_mlb[i] = 0;
        for (uint32_t i = threadIdx.x; i < 2 * mw + 1; i += blockDim.x) s_full[i] = 0;   // and s_np
        const uint32_t len[2] = {min(total, Vn), total > Vn ? total - Vn : 0u};
        const uint32_t first[2] = {s0, s0 + Vn}, w0[2] = {s0 / W, (s0 + Vn) / W};   // first samples, first windows
        float2 x[16];
        for (uint32_t c0 = 0; c0 < C; c0 += nh) {
            const uint32_t c = c0 + h;
            if (c0 + (h & ~1u) >= C) continue;   // the whole warp
            const bool on = c < C;
            const float* vr = P.V + (uint64_t)(on ? c : 0u) * d.N;
            float e = 0.f;
#pragma unroll
            for (uint32_t m = 0; m < 16; ++m) {
                const uint64_t ja = (uint64_t)first[0] + l + 16 * m, jb = ja + Vn;
                x[m].x = (on && ja < d.N) ? vr[ja] : 0.f;
                x[m].y = (on && len[1] > 0 && jb < d.N) ? vr[jb] : 0.f;
                e = fmaf(x[m].x, x[m].x, fmaf(x[m].y, x[m].y, e));
            }
            e = half_sum(e);
            if (on && l == 0) nz[c] = sqrtf(e) * 1.0001f;
            fft_channel(x, on ? zs + (size_t)c * 128 : reinterpret_cast<float4*>(xbuf + (size_t)h * kFft), tw, l);
        }
        FftAhead A;
        fft_fetch(P.F, C, h < M ? h : 0u, h < M, l, A);
        __syncthreads();
        // samples s with s + W < N have a likelihood, the others are 0 (binary_pursuit.cl:281-284)
        uint32_t lv[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            const uint64_t end = (uint64_t)d.N - W;
            lv[w] = first[w] < end ? (uint32_t)min((uint64_t)len[w], end - first[w]) : 0u;
        }
        for (uint32_t t0 = 0; t0 + (h & ~1u) < M; t0 += nh) {
            const uint32_t t = t0 + h;
            const bool on = t < M;
            const uint32_t tt = on ? t : 0u;
            const uint32_t cnt = A.cnt, cl = A.cl;
            const float tn = l < cnt ? P.tnorm[(size_t)tt * C + cl] : 0.f;
            fft_correlate(P.F, C, tt, A, t + nh, t + nh < M, zs, xbuf + (size_t)h * kFft, tw, l, x);
            float a = l < cnt ? tn * nz[cl] : 0.f;   // sum over the template's channels of |T_c| |z_c|
            for (uint32_t i = l + 16; i < cnt; i += 16) {
                const uint32_t c = P.F.clist[(size_t)tt * C + i];
                a = fmaf(P.tnorm[(size_t)tt * C + c], nz[c], a);
            }
            a = half_sum(a);
            const float4 tp = tpar[tt];
            // 1e-35: the products' own granularity where everything is tiny
            const float bd = tp.y * a + tp.z + (a > 0.f ? 1e-35f : 0.f);
            if (on && l == 0) tpar[t].w = bd;
            float* Lt = P.L + (uint64_t)tt * d.N;
            uint32_t can = 0;   // bits 0..15: outputs of the first stretch that can be positive, 16..31: of the second
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) {
                const uint32_t i = 16 * q + l;
                x[q].x += tp.x;
                x[q].y += tp.x;
                if (on && i < len[0]) Lt[first[0] + i] = i < lv[0] ? x[q].x : 0.f;
                if (on && i < len[1]) Lt[first[1] + i] = i < lv[1] ? x[q].y : 0.f;
                if (on && i < lv[0] && !(x[q].x + bd <= 0.f)) can |= 1u << q;
                if (on && i < lv[1] && !(x[q].y + bd <= 0.f)) can |= 0x10000u << q;
            }
            uint32_t any = __reduce_or_sync(0xffffffffu, can);
            if (any == 0u) continue;
            // the outputs through shared memory, so that the loop over the few that can be
            // positive is not unrolled over all
            float2* buf = xbuf + (size_t)h * kFft + l;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) buf[16 * q] = x[q];
#pragma unroll 1
            for (; any; any &= any - 1) {
                const uint32_t q2 = __ffs(any) - 1, w = q2 >> 4, i = 16 * (q2 & 15u) + l;
                const uint32_t s = (w ? first[1] : first[0]) + i;
                const float2 xv = buf[i - l];
                const float v = w ? xv.y : xv.x;
                const bool mine = (can >> q2) & 1u;
                const bool certain = mine && v - bd > 0.f;
                if (certain) {
                    const uint32_t ws = s / W;
                    int* slot = &s_mlb[w * P.wslots + ws - (w ? w0[1] : w0[0])];
                    atomicMax(slot, __float_as_int(v - bd));
                    if (!(v + bd >= __int_as_float(*(volatile int*)slot))) {
                        P.wflag[(uint64_t)ws * M + t] = 1;   // another sample of the window is larger
                    } else {
                        const uint32_t at = atomicAdd(s_np, 1u);
                        if (at < kPosCap) plist[at] = make_uint2((t << 9) | (w << 8) | i, __float_as_uint(v));
                        else atomicOr(&s_full[w * mw + (t >> 5)], 1u << (t & 31u));
                    }
                }
                const bool need = mine && !certain;
                if (__any_sync(0xffffffffu, need)) queue_samples(P, need, tt, s);
            }
            __syncwarp();
        }
        __syncthreads();   // the span's positives and lower bounds
        const uint32_t np = min(*s_np, kPosCap);
        for (uint32_t e = threadIdx.x; e < np; e += blockDim.x) {
            const uint2 g = plist[e];
            const uint32_t t = g.x >> 9, w = (g.x >> 8) & 1u, s = (w ? first[1] : first[0]) + (g.x & 255u);
            settle_positive(P, t, s, __uint_as_float(g.y), tpar[t].w,
                            __int_as_float(s_mlb[w * P.wslots + s / W - (w ? w0[1] : w0[0])]));
        }
        if (*s_np > kPosCap) {   // the list ran over: look at the stored estimates of the templates concerned
            for (uint32_t e = warp; e < 2 * M; e += blockDim.x >> 5) {
                const uint32_t w = e >= M ? 1u : 0u, t = e - w * M;
                if (!((s_full[w * mw + (t >> 5)] >> (t & 31u)) & 1u)) continue;
                const float bd = tpar[t].w;
                for (uint32_t i = lane; i < (w ? lv[1] : lv[0]); i += 32) {
                    const uint32_t s = (w ? first[1] : first[0]) + i;
                    const float v = P.L[(uint64_t)t * d.N + s];
                    if (v - bd > 0.f)
                        settle_positive(P, t, s, v, bd,
                                        __int_as_float(s_mlb[w * P.wslots + s / W - (w ? w0[1] : w0[0])]));
                }
            }
        }
        for (uint32_t i = threadIdx.x; i < 2 * P.wslots; i += blockDim.x)
            if (s_mlb[i] > 0) {
                const uint32_t w = i >= P.wslots ? 1u : 0u;
                P.wpos[(w ? w0[1] : w0[0]) + (i - w * P.wslots)] = 1;
            }
    }
}

// Spans of the listed windows: each run of consecutive windows, cut at multiples of
// kRunMost windows, into spans of at most 2 Vn samples; the windows' keys and flags
// are cleared.  The spans' order does not matter: a span's results are its own.
constexpr uint32_t kRunMost = 64;

__global__ void lik_units_kernel(Dims d, const uint32_t* __restrict__ list, uint32_t nlist, uint2* units,
                                 DevStatus* status, unsigned long long* wkey, uint8_t* wpos, uint8_t* wflag)
{
    const uint32_t span = 2 * lik_stretch(d.W), at = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (uint32_t k = at; k < nlist; k += step) {
        const uint32_t id = list[k];
        if ((uint64_t)id * d.W >= d.N) continue;
        wkey[id] = 0ull;
        wpos[id] = 0;
        if (k > 0 && list[k - 1] + 1 == id && id % kRunMost != 0) continue;
        uint32_t n = 1;
        while (k + n < nlist && list[k + n] == id + n && (id + n) % kRunMost != 0 && (uint64_t)(id + n) * d.W < d.N) ++n;
        const uint32_t s0 = id * d.W;
        const uint32_t len = (uint32_t)(min((uint64_t)(id + n) * d.W, (uint64_t)d.N) - s0);
        const uint32_t nu = (len + span - 1) / span;
        const uint32_t base = atomicAdd(&status->n_units, nu);
        for (uint32_t i = 0; i < nu; ++i) units[base + i] = make_uint2(s0 + i * span, min(span, len - i * span));
    }
    const uint64_t bytes = (uint64_t)nlist * d.M;
    for (uint64_t e = at; e < bytes; e += step) {
        const uint32_t id = list[e / d.M];
        if ((uint64_t)id * d.W < d.N) wflag[(uint64_t)id * d.M + e % d.M] = 0;
    }
}

// Half-warps per CTA and resident CTAs: the most useful half-warps per SM, counting
// the idle ones of the last round over the channels and over the templates (a
// template's product and inverse transform cost about 2.5 forward transforms).
struct FftShape {
    uint32_t nh = 0;
    uint32_t per_sm = 0;
    size_t smem = 0;
};

FftShape fft_shape(uint32_t C, uint32_t M, size_t extra)
{
    FftShape best;
    double top = 0.0;
    for (uint32_t nh : {8u, 16u, 32u}) {
        const size_t smem = (size_t)(C + nh + 1) * kFft * sizeof(float2) + extra;
        if (smem > kFftSmemMost) continue;
        const uint32_t regs = nh == 32 ? 128u : (nh == 16 ? 80u : 96u);   // as the launch bounds below allow
        const uint32_t per_sm = (uint32_t)std::min<size_t>((227 * 1024) / (smem + 1024), 65536 / (regs * nh * 16));
        if (per_sm == 0) continue;
        const double rounds = (double)((C + nh - 1) / nh) + 2.5 * ((M + nh - 1) / nh);
        const double useful = ((double)C + 2.5 * M) / (rounds * nh);
        const double score = useful * std::min<uint32_t>(per_sm * nh, 48);
        if (score > top) {
            top = score;
            best.nh = nh;
            best.per_sm = per_sm;
            best.smem = smem;
        }
    }
    return best;
}

}  // namespace

// The likelihood's extra shared memory behind the spectra and exchange buffers.
static size_t lik_extra(const Dims& d)
{
    return (size_t)d.M * 16 + kPosCap * 8 + ((size_t)d.C + 2 * (d.W ? lik_slots(d.W) : 0) + 2 * ((d.M + 31) / 32) + 1) * 4;
}

size_t fft_spectra_bytes(const Dims& d)
{
    const uint64_t b = (uint64_t)d.M * d.C * 128 * sizeof(float4);
    return (d.W <= 128 && d.C <= 256 && b <= kSpecMost && d.M < (1u << 22) &&
            fft_shape(d.C, d.M, lik_extra(d)).nh > 0) ? (size_t)b : 0;
}

bool fft_windows_supported(const Dims& d)
{
    return fft_spectra_bytes(d) > 0 && d.W + std::min(d.S, d.W - 1) <= kFft;
}

static FftTables fft_tables(const Work& w)
{
    const Layout& L = *w.lay;
    return FftTables{w.at<float4>(L.off_spec), w.at<uint8_t>(L.off_clist), w.at<uint32_t>(L.off_ccnt),
                     w.at<float2>(L.off_tw)};
}

int launch_template_info(const Dims& d, const Work& w, const float* T, cudaStream_t st, bool spectra)
{
    const Layout& L = *w.lay;
    count_launch();
    template_info_kernel<<<std::min<uint32_t>((d.M + 3) / 4, 148 * 8), 128, 0, st>>>(
        d, T, w.at<uint8_t>(L.off_clist), w.at<uint32_t>(L.off_ccnt), w.at<float>(L.off_tnorm),
        w.at<unsigned long long>(L.off_tchm), w.at<float>(L.off_tpad), w.at<float2>(L.off_lbnd));
    if (spectra && fft_spectra_bytes(d) > 0) {
        count_launch();
        spectra_kernel<<<d.M * d.C, kFft, 0, st>>>(d, T, w.at<uint8_t>(L.off_clist), w.at<uint32_t>(L.off_ccnt),
                                                   w.at<float4>(L.off_spec), w.at<float2>(L.off_tw));
    }
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

// The pursuit's likelihood by transforms: wherever they apply, unless the caller asked
// for the tensor-core kernel's launch shapes.  (The stand-alone fbp_likelihood keeps
// the tensor cores.)
bool fft_likelihood_chosen(const Dims& d)
{
    const fbp_tuning& tu = tuning();
    if (tu.lik_tiles || tu.lik_group || tu.lik_stages || tu.lik_epi) return false;   // the tensor-core kernel's shapes
    return fft_spectra_bytes(d) > 0;
}

uint64_t fft_span(const Dims& d) { return 2ull * lik_stretch(d.W); }

int launch_likelihood_fft(const Dims& d, const Work& w, const float* V, const float* T, const float* bias,
                          const uint32_t* list, uint32_t nlist, float* Lk, cudaStream_t st, uint64_t span0,
                          uint64_t span_count)
{
    if (nlist == 0) return FBP_OK;
    const Layout& L = *w.lay;
    const uint64_t span = fft_span(d), spans = ((uint64_t)d.N + span - 1) / span;
    const bool all = nlist == d.nw;
    if (all && span0 >= spans) return FBP_OK;
    LikFft P;
    P.d = d;
    P.F = fft_tables(w);
    P.V = V;
    P.T = T;
    P.bias = bias;
    P.tnorm = w.at<float>(L.off_tnorm);
    P.lbnd = w.at<float2>(L.off_lbnd);
    P.units = all ? nullptr : w.at<uint2>(L.off_units);
    P.n_spans = all ? (uint32_t)std::min<uint64_t>(span_count, spans - span0) : 0u;
    P.span0 = span0;
    P.L = Lk;
    P.fix = w.at<unsigned long long>(L.off_fix);
    P.fix_cap = (uint32_t)L.n_fix_cap;
    P.status = w.status();
    P.wkey = w.at<unsigned long long>(L.off_wkey);
    P.wpos = w.at<uint8_t>(L.off_wpos);
    P.wflag = w.at<uint8_t>(L.off_wflag);
    P.wslots = lik_slots(d.W);
    if (all) {
        if (span0 == 0)   // window keys, positive flags, estimate flags
            FBP_CUDA(cudaMemsetAsync(P.wkey, 0, L.off_wflag + L.nw * L.M - L.off_wkey, st));
        else              // a later range of the first pass: its own queue
            FBP_CUDA(cudaMemsetAsync(&w.status()->n_fix, 0, 4, st));
    } else {
        count_launch();
        lik_units_kernel<<<std::min<uint32_t>((nlist + 127) / 128, 148 * 8), 128, 0, st>>>(
            d, list, nlist, w.at<uint2>(L.off_units), w.status(), P.wkey, P.wpos, P.wflag);
    }
    const FftShape s = fft_shape(d.C, d.M, lik_extra(d));
    const uint32_t grid = std::min<uint32_t>(all ? P.n_spans : nlist, 148u * s.per_sm);
    count_launch();
    {
        KScope ks(&fbp_chunk_stats::ms_lik_tc, st);
#define FBP_LF(MAXT, MINB)                                              FBP_CUDA(allow_max_dyn_smem(lik_fft_kernel<MAXT, MINB>));           lik_fft_kernel<MAXT, MINB><<<grid, 16 * s.nh, s.smem, st>>>(P)
        if (s.nh <= 8) {
            FBP_LF(128, 5);
        } else if (s.nh <= 16) {
            FBP_LF(256, 3);
        } else {
            FBP_LF(512, 1);
        }
#undef FBP_LF
        FBP_CUDA(cudaGetLastError());
    }
    return launch_fixup(d, w, V, T, bias, Lk, true, st);
}

int launch_window_corr(const Dims& d, const Work& w, const float* V, const float* theta, const float2* Et,
                       uint32_t k0, uint32_t kc, float* G, float* vc2, float* z2, cudaStream_t st)
{
    const FftShape s = fft_shape(d.C, d.M, 0);
    const uint32_t grid = std::min<uint32_t>((kc + 1) / 2, 148u * s.per_sm);
    const FftTables F = fft_tables(w);
    count_launch();
#define FBP_WC(MAXT, MINB)                                                                                     \
    FBP_CUDA(allow_max_dyn_smem(window_corr_kernel<MAXT, MINB>));                                              \
    window_corr_kernel<MAXT, MINB><<<grid, 16 * s.nh, s.smem, st>>>(d, F, V, w.L(), theta, Et, w.flag(),       \
                                                                    w.status(), w.best_lab(), w.best_idx(),    \
                                                                    k0, kc, G, vc2, z2)
    if (s.nh <= 8) {
        FBP_WC(128, 5);
    } else if (s.nh <= 16) {
        FBP_WC(256, 3);
    } else {
        FBP_WC(512, 1);
    }
#undef FBP_WC
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

}  // namespace fbp
