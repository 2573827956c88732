// corr_fft.cu -- template correlations by 256-point transforms (fft256.cuh):
// the partial correlations of the overlap recheck.
//
// A template spans W samples on a few channels; correlating it with a window at
// every shift directly takes W multiply-adds per shift, channel and template.  By
// transforms the window's channels are transformed once, and each template costs
// one product per frequency and channel and one inverse transform.
#include <algorithm>

#include "fft256.cuh"

namespace fbp {
namespace {

constexpr size_t kFftSmemMost = 222 * 1024;   // dynamic shared memory of a CTA
constexpr size_t kSpecMost = 2ull << 30;      // bytes of template spectra

// Spectra, channel lists and the twiddle table, one CTA per (template, channel).
__global__ void __launch_bounds__(kFft) spectra_kernel(Dims d, const float* __restrict__ T, float4* spec, float2* tw)
{
    __shared__ double2 w[kFft];   // e^(-2 pi i k / 256)
    __shared__ float x[128];
    const uint32_t t = blockIdx.x / d.C, c = blockIdx.x % d.C, k = threadIdx.x;
    bool nz = false;
    if (k < d.W) {
        x[k] = T[((uint64_t)t * d.C + c) * d.W + k];
        nz = x[k] != 0.f;
    }
    const bool any = __syncthreads_or(nz) != 0;
    if (!any && blockIdx.x != 0) return;
    double sn, cs;
    sincospi(-2.0 * k / kFft, &sn, &cs);
    w[k] = make_double2(cs, sn);
    if (blockIdx.x == 0) {   // twiddles e^(2 pi i l r / 256) at r * 16 + l
        sincospi(2.0 * ((k & 15u) * (k >> 4)) / kFft, &sn, &cs);
        tw[k] = make_float2((float)cs, (float)sn);
    }
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

__global__ void channel_list_kernel(Dims d, const float* __restrict__ T, uint8_t* clist, uint32_t* ccnt)
{
    const uint32_t lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    for (uint32_t t = blockIdx.x * wpb + (threadIdx.x >> 5); t < d.M; t += gridDim.x * wpb) {
        uint32_t n = 0;
        for (uint32_t c = 0; c < d.C; ++c) {
            const float* r = T + ((uint64_t)t * d.C + c) * d.W;
            bool nz = false;
            for (uint32_t j = lane; j < d.W; j += 32) nz |= r[j] != 0.f;
            if (!__any_sync(0xffffffffu, nz)) continue;
            if (lane == 0) clist[(size_t)t * d.C + n] = (uint8_t)c;
            ++n;
        }
        if (lane == 0) ccnt[t] = n;
    }
}

// Partial correlations of flagged windows (see overlap_fast.cu):
//     G[k][t][b] = X_t(b) - 0.5 Et[t][b],   X_t(b) = sum_cj T[t][c][j - (b - S)] v[c][j]
// over the window's W samples, and the window's energy per channel, vc2[k][c].  A CTA
// takes two windows at a time (kk = 2 u, 2 u + 1 of the batch) as one complex signal:
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
    float* vc2)
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
    const uint32_t nflag = status->n_flag;
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
            if (on && l == 0) {
                if (2 * u < live) vc2[(size_t)(2 * u) * d.C + c] = ea;
                if (2 * u + 1 < live) vc2[(size_t)(2 * u + 1) * d.C + c] = eb;
            }
            // an idle half-warp of the last channels exchanges through a spare buffer
            fft_channel(x, on ? zs + (size_t)c * 128 : reinterpret_cast<float4*>(xbuf + (size_t)h * kFft), tw, l);
        }
        __syncthreads();
        float* Ga = G + (uint64_t)(2 * u) * M * S2;
        float* Gb = Ga + (uint64_t)M * S2;
        for (uint32_t t0 = 0; t0 + (h & ~1u) < M; t0 += nh) {
            const uint32_t t = t0 + h;
            const bool on = t < M;
            fft_correlate(F, d.C, on ? t : 0u, on, zs, xbuf + (size_t)h * kFft, tw, l, x);
            if (!on) continue;
            if (l == 0) macs += 4ull * kFft * F.ccnt[t];
            const float2* et = Et + (uint64_t)t * S2;
#pragma unroll
            for (uint32_t q = 0; q < 16; ++q) {
                const uint32_t n = 16 * q + l;   // shift n, or n - 256
                uint32_t b = 0xFFFFFFFFu;
                if (n <= Sw) b = n + S;
                else if (n + Sw >= kFft) b = n + S - kFft;
                if (b == 0xFFFFFFFFu) continue;
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

size_t fft_spectra_bytes(const Dims& d)
{
    const uint64_t b = (uint64_t)d.M * d.C * 128 * sizeof(float4);
    return (d.W <= 128 && d.C <= 256 && b <= kSpecMost && fft_shape(d.C, d.M, 0).nh > 0) ? (size_t)b : 0;
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

int launch_fft_templates(const Dims& d, const Work& w, const float* T, cudaStream_t st)
{
    if (fft_spectra_bytes(d) == 0) return FBP_OK;
    const Layout& L = *w.lay;
    count_launch(2);
    spectra_kernel<<<d.M * d.C, kFft, 0, st>>>(d, T, w.at<float4>(L.off_spec), w.at<float2>(L.off_tw));
    channel_list_kernel<<<std::min<uint32_t>((d.M + 3) / 4, 148 * 8), 128, 0, st>>>(d, T, w.at<uint8_t>(L.off_clist),
                                                                                   w.at<uint32_t>(L.off_ccnt));
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

int launch_window_corr(const Dims& d, const Work& w, const float* V, const float* theta, const float2* Et,
                       uint32_t k0, uint32_t kc, float* G, float* vc2, cudaStream_t st)
{
    const FftShape s = fft_shape(d.C, d.M, 0);
    const uint32_t grid = std::min<uint32_t>((kc + 1) / 2, 148u * s.per_sm);
    const FftTables F = fft_tables(w);
    count_launch();
#define FBP_WC(MAXT, MINB)                                                                                     \
    FBP_CUDA(allow_max_dyn_smem(window_corr_kernel<MAXT, MINB>));                                              \
    window_corr_kernel<MAXT, MINB><<<grid, 16 * s.nh, s.smem, st>>>(d, F, V, w.L(), theta, Et, w.flag(),       \
                                                                    w.status(), w.best_lab(), w.best_idx(),    \
                                                                    k0, kc, G, vc2)
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
