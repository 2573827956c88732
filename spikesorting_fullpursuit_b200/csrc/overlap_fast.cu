// overlap_fast.cu -- overlap recheck by screening, with exact results.
//
// The reference scores every item (a, t, b) of a flagged window
// (overlap_recheck_indices, binary_pursuit.cl:444-654) with C*W sequential
// float operations.  Its value expands as
//     v(a,t,b) = G_f(a) + G_t(b) - X_ft(a,b)
//     G_x(s)   = sum_cj X_s[c,j] v[c,j] - 0.5 sum_cj X_s[c,j]^2   (X_s: template x
//                shifted by s-S and cut to the window)
//     X_ft     = sum_cj F_a[c,j] T_b[c,j]
// G is a partial correlation of every template with the window (computed per
// window), X_ft depends only on the template pair and the two shifts (a table
// built once per call).  |v_ref - estimate| is bounded rigorously by a margin
// per window and template pair (pair_margin).  Only items whose interval can
// reach the best lower bound (and the window's seed likelihood) are scored
// exactly in the reference's float order; the winner key -- value, then
// work-group, then tree slot -- is therefore the reference's.
#include <algorithm>
#include <vector>

#include "fft256.cuh"

namespace fbp {
namespace {

__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }

// Truncated energies of template t (one CTA): E(x) = sum over the template samples
// u that land inside the window at shift x, u in [S-x, S-x+W) and [0, W), as
// (E, sqrt(E)), each rounded up (partial correlations), and their maxima over the
// shifts, maxs[t] = sqrt(E), maxs[M + t] = E (screening bound).
__global__ void __launch_bounds__(128) energy_table_kernel(Dims d, const float* __restrict__ T, float2* Et, float* maxs)
{
    extern __shared__ double cum[];   // [W + 1] running energy over the taps
    __shared__ int s_me, s_ms;
    const uint32_t t = blockIdx.x, S2 = 2 * d.S + 1, W = d.W;
    if (threadIdx.x == 0) { cum[0] = 0.0; s_me = 0; s_ms = 0; }
    for (uint32_t u = threadIdx.x; u < W; u += blockDim.x) {
        double e = 0.0;
        for (uint32_t c = 0; c < d.C; ++c) {
            const double v = T[((uint64_t)t * d.C + c) * W + u];
            e = fma(v, v, e);
        }
        cum[u + 1] = e;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (uint32_t u = 1; u <= W; ++u) cum[u] += cum[u - 1];
    __syncthreads();
    float me = 0.f, ms = 0.f;
    for (uint32_t x = threadIdx.x; x < S2; x += blockDim.x) {
        const int lo = max(0, (int)d.S - (int)x), hi = min((int)W, (int)d.S - (int)x + (int)W);
        // the difference of two running sums is off by at most 2 W 2^-53 of the whole energy
        const double e = hi > lo ? (cum[hi] - cum[lo]) * (1.0 + 1e-12) + cum[W] * 1e-12 : 0.0;
        const float ef = __double2float_ru(e), es = __double2float_ru(sqrt(e) * (1.0 + 1e-12));
        Et[(uint64_t)t * S2 + x] = make_float2(ef, es);
        me = fmaxf(me, ef);
        ms = fmaxf(ms, es);
    }
    atomicMax(&s_me, __float_as_int(me));   // both >= 0
    atomicMax(&s_ms, __float_as_int(ms));
    __syncthreads();
    if (threadIdx.x == 0) {
        maxs[t] = __int_as_float(s_ms);
        maxs[d.M + t] = __int_as_float(s_me);
    }
}

// largest value of the warp's lanes, NaN ignored; volatile, since all lanes have to reach it
// and some uses are by one lane only: plain asm may be moved into such a branch
__device__ __forceinline__ float warp_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Pair cross terms X_ft(a, b) for |a-b| <= W, one CTA per (f, t), stored as
// XT[f][t][a][b] and transposed as XTT[f][t][b][a]: products
// P_delta[u] = sum_c F[c,u] T[c,u+delta] in double, prefix sums over u, then
// X_ft(a, b) = Q_delta[hi] - Q_delta[lo] with delta = a-b.  Pairs without a shared
// channel have X == 0: their table is never read and stays unwritten.  Also the
// bounds over whole chunks of 32 shifts, XC[f][a][t][ch] = max over b of the chunk,
// |a-b| <= W, of -X_ft(a, b) (-inf if there is none) and XCT[f][t][b][ch] over a, and
// max -X (at least 0) per pair.  32 lags at a time: a lag is a lane, so that a warp
// writes 32 consecutive shifts of a row (with the row index on the lanes every 4-byte
// store was a sector of its own: 64 channels x 200 templates about 12 ms of a call).
//
// With few pairs the groups of lags are split over gridDim.y CTAs a pair, and the
// bounds, which need whole rows, follow in a launch of their own: 4 channels, 6 templates,
// 201 x 201 shifts 177 us by one CTA a pair, 17 + 12 us so.  With
// many pairs one CTA does both, the rows then still being in the L1 and L2.
constexpr int kCrossThreads = 256;

// XC, XCT and max -X of pair `p`, rows `first`, first + step, ... (a warp a row)
__device__ __forceinline__ void cross_bounds(const Dims& d, uint32_t p, uint32_t first, uint32_t step,
                                             const float* XT, const float* XTT, float* XC, float* XCT, int* neg_bits)
{
    const uint32_t f = p / d.M, t = p % d.M, lane = threadIdx.x & 31;
    const uint32_t S2 = 2 * d.S + 1, nch = (S2 + 31) / 32;
    float neg = 0.f;
    for (uint32_t e = first; e < 2 * S2; e += step) {
        const uint32_t y = e >> 1;
        const float* row = ((e & 1u) ? XTT : XT) + (uint64_t)p * S2 * S2 + (uint64_t)y * S2;
        float* out = (e & 1u) ? XCT + ((uint64_t)p * S2 + y) * nch : XC + (((uint64_t)f * S2 + y) * d.M + t) * nch;
#pragma unroll 4
        for (uint32_t ch = 0; ch < nch; ++ch) {
            const uint32_t x = ch * 32 + lane;
            const bool in = x < S2 && x + d.W >= y && x <= y + d.W;
            const float m = warp_max(in ? -row[x] : -INFINITY);
            if (lane == 0) out[ch] = m;
            neg = fmaxf(neg, m);
        }
    }
    if (lane == 0) atomicMax(neg_bits, __float_as_int(neg));   // neg >= 0
}

__global__ void __launch_bounds__(kCrossThreads) cross_bound_kernel(Dims d,
                                                                    const unsigned long long* __restrict__ chmask,
                                                                    const float* XT, const float* XTT, float* XC,
                                                                    float* XCT, float* max_negx)
{
    const uint32_t p = blockIdx.x, warps = kCrossThreads / 32;
    if ((chmask[p / d.M] & chmask[p % d.M]) == 0ull) return;
    cross_bounds(d, p, blockIdx.y * warps + (threadIdx.x >> 5), gridDim.y * warps, XT, XTT, XC, XCT,
                 reinterpret_cast<int*>(max_negx) + p);
}

__global__ void __launch_bounds__(kCrossThreads) cross_table_kernel(Dims d, const float* __restrict__ T,
                                                                    const unsigned long long* __restrict__ chmask,
                                                                    int lags, float* XT, float* XTT, float* XC,
                                                                    float* XCT, float* max_negx)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ int s_neg;
    const uint32_t f = blockIdx.x / d.M, t = blockIdx.x % d.M;
    const uint32_t S2 = 2 * d.S + 1, W = d.W, C = d.C;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = kCrossThreads / 32;
    const unsigned long long both = chmask[f] & chmask[t];   // all ones above 64 channels
    if (both == 0ull) {
        if (threadIdx.x == 0 && blockIdx.y == 0) max_negx[blockIdx.x] = 0.f;
        return;
    }
    const uint32_t pitch = (W + 1) | 1u;   // odd: the lags of a warp read different banks
    float* Fs = reinterpret_cast<float*>(smraw);
    float* Ts = Fs + C * W;
    double* Q = reinterpret_cast<double*>(Ts + C * W);  // [lags <= 32][pitch]; 8*C*W bytes in, aligned
    if (threadIdx.x == 0) s_neg = 0;
    for (uint32_t e = threadIdx.x; e < C * W; e += blockDim.x) {
        Fs[e] = T[(uint64_t)f * C * W + e];
        Ts[e] = T[(uint64_t)t * C * W + e];
    }
    __syncthreads();
    float* xt = XT + (uint64_t)blockIdx.x * S2 * S2;
    float* xtt = XTT + (uint64_t)blockIdx.x * S2 * S2;
    const int dmax = (int)min(W, 2 * d.S);
    for (int d0 = -dmax + (int)blockIdx.y * lags; d0 <= dmax; d0 += (int)gridDim.y * lags) {
        for (int li = warp; li < lags; li += nwarps) {
            const int delta = d0 + li;
            double* q = Q + li * pitch;
            double run = 0.0;   // prefix sums of a lag by a warp, 32 taps at a time
            if (lane == 0) q[0] = 0.0;
            for (uint32_t u0 = 0; u0 < W; u0 += 32) {
                const int u = (int)(u0 + lane);
                double acc = 0.0;
                if (u < (int)W && u + delta >= 0 && u + delta < (int)W && delta <= dmax) {
                    if (C <= 64)
                        for (unsigned long long m = both; m; m &= m - 1) {
                            const uint32_t c = __ffsll((long long)m) - 1;
                            acc = fma((double)Fs[c * W + u], (double)Ts[c * W + u + delta], acc);
                        }
                    else
                        for (uint32_t c = 0; c < C; ++c)
                            acc = fma((double)Fs[c * W + u], (double)Ts[c * W + u + delta], acc);
                }
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const double o = __shfl_up_sync(0xffffffffu, acc, off);
                    if ((int)lane >= off) acc += o;
                }
                acc += run;
                if (u < (int)W) q[u + 1] = acc;
                run = __shfl_sync(0xffffffffu, acc, 31);
            }
        }
        __syncthreads();
        const int delta = (int)lane < lags ? d0 + (int)lane : dmax + 1;
        for (int a = (int)warp; a < (int)S2; a += nwarps) {   // row a: shifts b = a - delta
            const int b = a - delta;
            if (delta > dmax || b < 0 || b >= (int)S2) continue;
            const int lo = max(max(0, -delta), (int)d.S - a);
            const int hi = min(min((int)W, (int)W - delta), (int)d.S - a + (int)W);
            xt[(uint64_t)a * S2 + b] = hi > lo ? (float)(Q[lane * pitch + hi] - Q[lane * pitch + lo]) : 0.f;
        }
        for (int b = (int)warp; b < (int)S2; b += nwarps) {   // row b of the transposed table: a = b + delta
            const int a = b + delta;
            if (delta > dmax || a < 0 || a >= (int)S2) continue;
            const int lo = max(max(0, -delta), (int)d.S - a);
            const int hi = min(min((int)W, (int)W - delta), (int)d.S - a + (int)W);
            xtt[(uint64_t)b * S2 + a] = hi > lo ? (float)(Q[lane * pitch + hi] - Q[lane * pitch + lo]) : 0.f;
        }
        __syncthreads();
    }
    if (gridDim.y > 1) {
        if (threadIdx.x == 0 && blockIdx.y == 0) max_negx[blockIdx.x] = 0.f;   // cross_bound_kernel raises it
        return;
    }
    cross_bounds(d, blockIdx.x, warp, nwarps, XT, XTT, XC, XCT, &s_neg);
    __syncthreads();
    if (threadIdx.x == 0) max_negx[blockIdx.x] = __int_as_float(s_neg);
}

// Template processing order of the direct partial correlations: sorted by the first
// non-zero channel so groups of neighbouring templates share channels.
__global__ void template_order_kernel(Dims d, const uint8_t* __restrict__ clist, const uint32_t* __restrict__ ccnt,
                                      uint32_t* perm)
{
    extern __shared__ uint32_t key[];
    for (uint32_t t = threadIdx.x; t < d.M; t += blockDim.x) key[t] = ccnt[t] ? clist[(size_t)t * d.C] : d.C;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (uint32_t t = 0; t < d.M; ++t) perm[t] = t;
        for (uint32_t i = 1; i < d.M; ++i) {  // stable insertion sort by key
            const uint32_t v = perm[i];
            int j = (int)i - 1;
            while (j >= 0 && key[perm[j]] > key[v]) { perm[j + 1] = perm[j]; --j; }
            perm[j + 1] = v;
        }
    }
}

__device__ __forceinline__ bool window_skipped(const Dims& d, const float* L, const float* theta, uint32_t f,
                                               uint32_t p)
{
    return L[(uint64_t)f * d.N + p] < theta[f] || (uint64_t)p >= (uint64_t)d.N - d.W;
}

// Partial correlations G[k][t][b] = X_t(b) - 0.5 Et[t][b] of every template
// with each flagged window (masked to [p, p+W)).  A CTA owns one group of Q
// templates (in perm order; only the group's union of non-zero channels is
// staged) and walks over the windows kPcWin at a time.  Lane = (window, shift
// sub-block): a warp covers 16 consecutive shifts of 8 windows, so the taps
// that can meet the window's W live samples form one range per warp (the
// zero triangle of the masked correlation is skipped), and each lane computes
// 4 consecutive shifts for the Q templates from aligned 16-byte strip loads.
// The strips keep their zero margins from one clearing; each window writes
// only its W live samples per channel (cp.async).  The sums are estimates:
// any order, FMA allowed.
constexpr int kPcR = 4;       // shifts per lane
constexpr int kPcWin = 8;     // windows per CTA iteration (lane bits 2..4)
constexpr int kPcPad = 20;    // zero margin around the live samples in a staged strip
constexpr int kPcMaxWarps = 12;   // two CTAs of 12 warps fit an SM at <= 80 registers

struct PcGeom {
    uint32_t Wp, Z, SLc, WS;  // padded taps; strip index of window sample 0; strip length; window stride
    int o;                    // shift b reads strip index b - o + j  (o = S - Z, a multiple of 4)
};

__host__ __device__ inline PcGeom pc_geom(const Dims& d, uint32_t Cu)
{
    PcGeom g;
    g.Wp = (d.W + 3) & ~3u;
    g.Z = kPcPad + (d.S & 3u);
    g.o = (int)d.S - (int)g.Z;
    g.SLc = (g.Z + d.W + kPcPad + 3) & ~3u;
    uint32_t ws = Cu * g.SLc;
    ws += (16u - ws % 32u + 32u) % 32u;   // windows 16 banks apart: a quarter-warp's two windows do not collide
    g.WS = ws;
    return g;
}

__host__ __device__ inline size_t pc_smem_bytes(const Dims& d, uint32_t Cu, int Q)
{
    const PcGeom g = pc_geom(d, Cu);
    return ((size_t)Q * Cu * g.Wp + (size_t)kPcWin * g.WS) * 4;
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src)
{
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(src) : "memory");
}

template <int Q>
__global__ void __launch_bounds__(kPcMaxWarps * 32, 2) partial_corr_kernel(
    Dims d, const float* __restrict__ V, const float* __restrict__ T, const float* __restrict__ L,
    const float* __restrict__ theta, const float2* __restrict__ Et, const uint32_t* __restrict__ perm,
    const unsigned long long* __restrict__ chmask, const uint32_t* __restrict__ flag, const DevStatus* status,
    const uint32_t* __restrict__ best_lab, const uint32_t* __restrict__ best_idx, uint32_t k0, uint32_t kc,
    float* G)
{
    extern __shared__ __align__(16) float sm[];
    __shared__ uint32_t chans[256];
    __shared__ uint32_t s_nch;
    __shared__ uint32_t s_p[kPcWin];
    __shared__ int s_ok[kPcWin];
    const uint32_t S2 = 2 * d.S + 1, W = d.W, M = d.M;
    const uint32_t g0 = blockIdx.y * Q;
    if (threadIdx.x == 0) {
        unsigned long long m = 0ull;
        for (uint32_t q = 0; q < Q; ++q)
            if (g0 + q < M) m |= chmask[perm[g0 + q]];
        uint32_t n = 0;
        for (uint32_t c = 0; c < d.C; ++c)
            if (c >= 64 || ((m >> c) & 1ull)) chans[n++] = c;
        s_nch = n;
    }
    __syncthreads();
    const uint32_t Cu = s_nch;
    const PcGeom gm = pc_geom(d, Cu);
    const uint32_t Wp = gm.Wp;
    float* Ts = sm;                                   // [Q][Cu][Wp]
    float* Vs = sm + (size_t)Q * Cu * Wp;              // [kPcWin][WS], row ci at ci * SLc
    for (uint32_t e = threadIdx.x; e < Q * Cu * Wp; e += blockDim.x) {
        const uint32_t q = e / (Cu * Wp), r = e - q * Cu * Wp, ci = r / Wp, j = r - ci * Wp;
        Ts[e] = (g0 + q < M && j < W) ? T[((uint64_t)perm[g0 + q] * d.C + chans[ci]) * W + j] : 0.f;
    }
    for (uint32_t e = threadIdx.x; e < kPcWin * gm.WS; e += blockDim.x) Vs[e] = 0.f;
    const uint32_t nflag = flagged_windows(status);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t wi = lane >> 2, bs = lane & 3;
    unsigned long long macs = 0;   // multiply-adds this thread does
    for (uint32_t base = blockIdx.x * kPcWin; base < kc; base += gridDim.x * kPcWin) {
        __syncthreads();
        if (threadIdx.x < kPcWin) {
            const uint32_t kk = base + threadIdx.x;
            int ok = 0;
            uint32_t p = 0;
            if (kk < kc && k0 + kk < nflag) {
                const uint32_t id = flag[k0 + kk];
                const uint32_t f = best_lab[id];
                p = best_idx[id];
                ok = !window_skipped(d, L, theta, f, p);
            }
            s_ok[threadIdx.x] = ok;
            s_p[threadIdx.x] = p;
        }
        __syncthreads();
        for (uint32_t r = warp; r < kPcWin * Cu; r += nwarps) {
            const uint32_t w = r / Cu, ci = r - w * Cu;
            if (!s_ok[w]) continue;
            const float* src = V + (uint64_t)chans[ci] * d.N + s_p[w];
            float* dst = Vs + (size_t)w * gm.WS + (size_t)ci * gm.SLc + gm.Z;
            for (uint32_t j = lane; j < W; j += 32) cp_async4(dst + j, src + j);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (!s_ok[wi]) continue;
        float* Gk = G + (uint64_t)(base + wi) * M * S2;
        const float* vw = Vs + (size_t)wi * gm.WS;
        for (uint32_t bw = warp * 16; bw < S2; bw += nwarps * 16) {
            const uint32_t b0 = bw + kPcR * bs;
            int jlo = (int)d.S - (int)bw - 15;
            jlo = jlo < 0 ? 0 : (jlo & ~3);
            int jhi = ((int)(d.S + W) - (int)bw + 3) & ~3;
            jhi = jhi > (int)Wp ? (int)Wp : jhi;
            float acc[Q][kPcR];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < kPcR; ++r) acc[q][r] = 0.f;
            const int vb = (int)b0 - gm.o;
            if (jhi > jlo) macs += (unsigned long long)Q * kPcR * (uint32_t)(jhi - jlo) * Cu;
            for (uint32_t ci = 0; ci < Cu; ++ci) {
                const float* vr = vw + (size_t)ci * gm.SLc;
                const float* tr = Ts + (size_t)ci * Wp;
                for (int j0 = jlo; j0 < jhi; j0 += 4) {
                    const float4 va = *reinterpret_cast<const float4*>(vr + vb + j0);
                    const float4 vc = *reinterpret_cast<const float4*>(vr + vb + j0 + 4);
                    const float v[8] = {va.x, va.y, va.z, va.w, vc.x, vc.y, vc.z, vc.w};
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const float4 t4 = *reinterpret_cast<const float4*>(tr + (size_t)q * Cu * Wp + j0);
#pragma unroll
                        for (int r = 0; r < kPcR; ++r) {
                            float a = acc[q][r];
                            a = fmaf(t4.x, v[r], a);
                            a = fmaf(t4.y, v[r + 1], a);
                            a = fmaf(t4.z, v[r + 2], a);
                            a = fmaf(t4.w, v[r + 3], a);
                            acc[q][r] = a;
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                if (g0 + q >= M) continue;
                const uint32_t t = perm[g0 + q];
#pragma unroll
                for (int r = 0; r < kPcR; ++r) {
                    const uint32_t bb = b0 + r;
                    if (bb < S2) Gk[(uint64_t)t * S2 + bb] = acc[q][r] - 0.5f * Et[(uint64_t)t * S2 + bb].x;
                }
            }
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) macs += __shfl_xor_sync(0xffffffffu, macs, off);
    if (lane == 0 && macs) atomicAdd(&const_cast<DevStatus*>(status)->pc_macs, macs);
}

// Exact pair likelihood in the reference's float order (binary_pursuit.cl:578-632),
// operands read from memory.
// Channels on which both templates are entirely zero are skipped: there the
// reference adds 0 * v and 0 * 0 terms, which leave its sums unchanged (acc
// starts at +0, so no step of the reference makes it -0 either).
__device__ float pair_exact_g(const Dims& d, const float* __restrict__ T, const float* __restrict__ V, uint32_t f,
                              uint32_t t, uint32_t p, uint32_t a, uint32_t b, unsigned long long chans)
{
    const int W = (int)d.W, fa = (int)d.S - (int)a, ta = (int)d.S - (int)b;
    const int jlo_f = max(0, -fa), jhi_f = min(W, W - fa), jlo_t = max(0, -ta), jhi_t = min(W, W - ta);
    float acc = 0.f;
    for (uint32_t c = 0; c < d.C; ++c) {
        if (c < 64 && !((chans >> c) & 1ull)) continue;
        const float* fr = T + ((uint64_t)f * d.C + c) * d.W + fa;
        const float* tr = T + ((uint64_t)t * d.C + c) * d.W + ta;
        const float* vr = V + (uint64_t)c * d.N + p;
        float ss = 0.f;
#pragma unroll 8
        for (int j = 0; j < W; ++j) {
            const float fv = (j >= jlo_f && j < jhi_f) ? __ldg(fr + j) : 0.f;
            const float tv = (j >= jlo_t && j < jhi_t) ? __ldg(tr + j) : 0.f;
            const float sv = fadd(fv, tv);
            ss = fadd(ss, fmul(sv, sv));
            acc = fadd(acc, fmul(sv, __ldg(vr + j)));
        }
        if (ss > 0.f) acc = fsub(acc, fmul(0.5f, ss));
    }
    return acc;
}

// the same, out of line
__device__ __noinline__ float pair_exact_call(const Dims d, const float* T, const float* V, uint32_t f, uint32_t t,
                                              uint32_t p, uint32_t a, uint32_t b, unsigned long long chans)
{
    return pair_exact_g(d, T, V, f, t, p, a, b, chans);
}

__device__ __forceinline__ uint32_t item_priority(uint64_t r, uint32_t WG, uint32_t lbits)
{
    const uint32_t g = (uint32_t)(r / WG), l = (uint32_t)(r % WG);
    const uint32_t br = lbits ? (__brev(l) >> (32 - lbits)) : 0u;
    return g * WG + br;
}

constexpr uint32_t kChunkCap = 512;    // chunks of 32 items kept in shared memory
constexpr uint32_t kRowCap = 768;      // rows (t, b) kept in shared memory
constexpr uint32_t kQueue = 64;        // chunks a warp keeps for evaluation
// Threads a window, and CTAs per SM.  A window alone takes its loads one after the
// other: with no more listed windows than kScrFewWindows, of which a part is flagged,
// the SMs are not full and 512 threads a window are faster (3 to 12 s of 4 to 12
// channels, up to 300 flagged windows a pass: 70 -> 44 us; 20 s of 64 channels 14.3 ->
// 12.5 ms a pursuit); many windows fill the SMs with 128 threads each, and a CTA of 512
// waits for its slowest warp at every barrier (512 for all, 300 s of 16 channels: 14.1
// -> 21.5 ms; the line at 2400, 5000 and 10000 windows: within 1% there, 12.6, 12.5 and
// 13.2 ms with 64 channels).
constexpr int kScrThreads = 128, kScrPerSm = 8;
constexpr int kScrWideThreads = 512, kScrWidePerSm = 2;
constexpr uint32_t kScrFewWindows = 5000;

struct ScreenArgs {
    Dims d;
    const float* V;
    const float* T;
    const float* L;
    const float* theta;
    const float* XT;
    const float* XTT;
    const float* XC;
    const float* XCT;
    const float* mx;        // [M][M] max -X, then [M] max sqrt(E), [M] max E
    const float* G;
    const float* vc2;       // [kc][C] window energies per channel, or null: from the voltage (direct correlations)
    const float* z2;        // [kc][C] energies of the signal pair transformed together
    uint32_t k0, kc;
    const uint32_t* flag;
    DevStatus* status;
    const uint32_t* best_lab;
    const uint32_t* best_idx;
    const float* best_lik;
    unsigned long long* keys;
    unsigned long long* gcand;
    uint32_t cand_cap;
    const unsigned long long* chmask;
    const uint32_t* order;
};

struct ScreenShared {
    int lb;              // largest lower bound, float bits (0: none above 0)
    uint32_t nA, top;    // shifts in A+, the place in alist of the largest G_f
    uint32_t nrows, nchunks, full;
    unsigned long long best;
};

__host__ __device__ inline uint32_t scr_chunks(uint32_t S2) { return (S2 + 31) / 32; }

// Shared-memory bytes of screen_kernel.
__host__ __device__ inline size_t screen_smem_bytes(uint32_t M, uint32_t S2, uint32_t C, int threads)
{
    const size_t nch = scr_chunks(S2);
    return (nch * 32 * 2 + (size_t)M * nch * 2 + (size_t)M * 4 + nch + C * 2 + kChunkCap * 3 + kRowCap * 2 +
            kQueue * 2 * (size_t)(threads / 32)) * 4 + 16;
}

// Bound of |estimate - reference float value| of every item (a, t, b) of a window
// with best template f, u = 2^-24, over the templates' whole energies E (at least any
// truncated one):
//     u 1.06 [ (U (W + 1) + W + 48) (A_f + A_t) + B_f + B_t ],
//     A_x = sqrt E_x |v|_x + E_x,  |v|_x the window's norm over template x's channels.
// The first part: the reference adds U (W + 1) terms one at a time, U the channels
// where f or t is not zero (elsewhere it adds exact zeros), W of each channel's
// energy, and the estimate's own few operations; |s v| <= |f v| + |t v|,
// s^2 <= 2 f^2 + 2 t^2.  B_x: the partial correlations -- by transforms
// (64 + 3 n_x) sqrt E_x |z|_x (fft256.cuh, z the pair of windows transformed
// together), directly n_x W sqrt E_x |v|_x.  An infinite margin (the window's energy
// overflows) keeps every item, NaN (a sample is not finite: so are the reference's
// values) none.
struct MarginPart {
    float a, b;   // A_x, B_x
};

__device__ __forceinline__ MarginPart margin_part(const ScreenArgs& P, uint32_t t, const float* ve, const float* ze)
{
    const Dims& d = P.d;
    float v2 = 0.f, z2 = 0.f;
    uint32_t n = 0;
    const unsigned long long m = P.chmask[t];
    for (uint32_t c = 0; c < d.C; ++c)
        if (d.C > 64 || ((m >> c) & 1ull)) {
            v2 += ve[c];
            z2 += ze[c];
            ++n;
        }
    const float se = P.mx[(size_t)d.M * d.M + t], e = P.mx[(size_t)d.M * d.M + d.M + t];
    const float nv = se > 0.f ? sqrtf(v2) * 1.001f : 0.f, nz = se > 0.f ? sqrtf(z2) * 1.001f : 0.f;
    MarginPart r;
    r.a = fmaf(se, nv, e);
    r.b = P.vc2 ? (kFftTerms + 3.f * n) * se * nz : (float)n * d.W * se * nv;
    return r;
}

__device__ __forceinline__ float pair_margin(const Dims& d, MarginPart f, MarginPart t, uint32_t U)
{
    return 1.06f / 16777216.f * (((float)U * (d.W + 1) + d.W + 48.f) * (f.a + t.a) + f.b + t.b);
}

// Screening of one flagged window per CTA.
//   rows, kind 0: (a in A+, t) -- a fixed, the lanes run over b (XT[f][t][a][:]);
//   rows, kind 1: (t, b) with L_t(b) > 0 -- b fixed, the lanes run over a not in A+
//                 (XTT[f][t][b][:]),
// A+ the in-bounds shifts with L_f > 0.  An item's interval is its estimate
// (G_f(a) + G_t(b)) - X +- margin.  A row is taken up while an upper bound (largest G
// of its variable shift, largest -X of the pair) reaches the seed and the lower bound
// so far, then those of its chunks of 32 items whose own bound (largest G and largest
// -X of the chunk) does, then their items, which raise the lower bound; the rows of
// the a with the largest G_f come first.  Chunks with an item that reaches the lower
// bound are kept, and their items listed for score_kernel in the end.
//
// 32 rows are tested at a time, one a lane; the chunks that pass are queued per warp
// and evaluated eight at a time, their loads in flight together.  About 270 (16
// channels x 40 templates) and 300 chunks (64 x 200) are evaluated per window, and 1 to
// 9 items of it reach the exact scoring.  Measured per pursuit, against whole rows
// scanned after staging G +- margin of every template and shift: 300 s of 16 channels
// 31.9 -> 14.5 ms, 20 s of 64 channels 37.4 -> 14.3 ms (and 8.5 M -> 0.16 M items
// scored exactly there, by the margin's count of non-zero channels).  Bounded by
// instruction issue and latency together: 49 % of the issue slots, 28 warps per SM.
template <int THREADS, int PER_SM>
__global__ void __launch_bounds__(THREADS, PER_SM) screen_kernel(const __grid_constant__ ScreenArgs P)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ ScreenShared sh;
    const Dims& d = P.d;
    const uint32_t S = d.S, W = d.W, M = d.M, C = d.C, S2 = 2 * S + 1, nch = scr_chunks(S2);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = THREADS / 32;
    const uint32_t full = 0xffffffffu, below = (1u << lane) - 1u;
    float* Gf = reinterpret_cast<float*>(smraw);                       // [nch * 32] G_f, -inf out of bounds
    uint32_t* alist = reinterpret_cast<uint32_t*>(Gf + nch * 32);      // [nch * 32] A+ in ascending order
    float* gch = reinterpret_cast<float*>(alist + nch * 32);           // [M][nch] largest G_t of a chunk
    uint32_t* pb = reinterpret_cast<uint32_t*>(gch + (size_t)M * nch); // [M][nch] shifts with L_t > 0
    float* gmax = reinterpret_cast<float*>(pb + (size_t)M * nch);      // [M] largest G_t
    float* nx = gmax + M;                                              // [M] largest -X_ft
    float* cst = nx + M;                                               // [M] margin of the pair (f, t)
    uint32_t* share = reinterpret_cast<uint32_t*>(cst + M);            // [M] f and t share a channel
    float* afch = reinterpret_cast<float*>(share + M);                 // [nch] largest G_f of a chunk, a not in A+
    float* ve = afch + nch;                                            // [C] window energies
    float* ze = ve + C;                                                // [C] pair energies
    uint32_t* chc = reinterpret_cast<uint32_t*>(ze + C);               // [kChunkCap] chunk << 23 | row (kind << 22 | t << 10 | y)
    float* chu = reinterpret_cast<float*>(chc + kChunkCap);            // [kChunkCap] upper bound of its items
    float* chg = chu + kChunkCap;                                      // [kChunkCap] the row's fixed G
    uint32_t* rowc = reinterpret_cast<uint32_t*>(chg + kChunkCap);     // [kRowCap] rows (t, b) that can reach the seed
    float* rowg = reinterpret_cast<float*>(rowc + kRowCap);            // [kRowCap] their G_t(b)
    uint32_t* qc = reinterpret_cast<uint32_t*>(rowg + kRowCap) + warp * kQueue;   // this warp's chunks to evaluate
    float* qg = reinterpret_cast<float*>(qc - warp * kQueue + nwarps * kQueue) + warp * kQueue;   // their rows' fixed G
    const uint64_t items = (uint64_t)S2 * S2 * M;
    const uint64_t slots = ((items - 1) / d.WG + 1) * d.WG;
    uint32_t lbits = 0;
    while ((1u << lbits) < d.WG) ++lbits;
    const uint32_t nflag = flagged_windows(P.status);
    const uint32_t live = nflag > P.k0 ? min(P.kc, nflag - P.k0) : 0u;
    uint32_t evals = 0;   // chunks evaluated by this warp
    for (uint32_t jo = blockIdx.x; jo < live; jo += gridDim.x) {
        const uint32_t kk = P.order[jo];
        const uint32_t id = P.flag[P.k0 + kk];
        const uint32_t f = P.best_lab[id], p = P.best_idx[id];
        if (window_skipped(d, P.L, P.theta, f, p)) continue;
        const float thr0 = fmaxf(P.best_lik[id], 0.f);   // the seed
        const float* Gk = P.G + (uint64_t)kk * M * S2;
        // in-bounds shifts x: x + p >= S and x + p < N - W + S
        const uint32_t xlo = p < S ? S - p : 0u;
        const uint32_t xhi = (uint32_t)min((uint64_t)S2, (uint64_t)d.N - W + S - p);
        __syncthreads();   // the previous window's shared state is read
        for (uint32_t c = threadIdx.x; P.vc2 != nullptr && c < C; c += blockDim.x) {
            ve[c] = P.vc2[(size_t)kk * C + c];
            ze[c] = P.z2[(size_t)kk * C + c];
        }
        for (uint32_t c = warp; P.vc2 == nullptr && c < C; c += nwarps) {
            float e = 0.f;
            for (uint32_t j = lane; j < W; j += 32) {
                const float v = P.V[(uint64_t)c * d.N + p + j];
                e = fmaf(v, v, e);
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) e += __shfl_xor_sync(full, e, off);
            if (lane == 0) {
                ve[c] = e;
                ze[c] = 0.f;
            }
        }
        // template f's shifts
        for (uint32_t ch = warp; ch < nch; ch += nwarps) {
            const uint32_t x = ch * 32 + lane;
            const bool in = x >= xlo && x < xhi;
            const float g = in ? Gk[(uint64_t)f * S2 + x] : -INFINITY;
            const bool pos = in && P.L[(uint64_t)f * d.N + p + x - S] > 0.f;
            const uint32_t bits = __ballot_sync(full, pos);
            const float m = warp_max(pos ? -INFINITY : g);
            Gf[x] = g;
            if (lane == 0) {
                pb[(size_t)f * nch + ch] = bits;
                afch[ch] = m;
            }
        }
        if (threadIdx.x == 0) {
            sh.lb = 0;
            sh.nrows = 0;
            sh.nchunks = 0;
            sh.full = 0;
            sh.best = 0ull;
        }
        __syncthreads();
        {
            const unsigned long long mf = P.chmask[f];
            const MarginPart pf = margin_part(P, f, ve, ze);
            for (uint32_t t = threadIdx.x; t < M; t += blockDim.x) {
                const unsigned long long mt = P.chmask[t];
                const uint32_t U = C > 64 ? C : (uint32_t)__popcll((long long)(mf | mt));
                cst[t] = pair_margin(d, pf, margin_part(P, t, ve, ze), U);
                nx[t] = P.mx[(uint64_t)f * M + t];
                share[t] = (mf & mt) != 0ull;
            }
        }
        if (warp == nwarps - 1) {   // A+ in ascending order, and the a in A+ with the largest G_f
            uint32_t n = 0, ba = 0;
            float bg = -INFINITY;
            for (uint32_t ch = 0; ch < nch; ++ch) {
                const uint32_t bits = pb[(size_t)f * nch + ch];
                if ((bits >> lane) & 1u) {
                    const uint32_t at = n + __popc(bits & below);
                    alist[at] = ch * 32 + lane;
                    if (Gf[ch * 32 + lane] > bg) {
                        bg = Gf[ch * 32 + lane];
                        ba = at;
                    }
                }
                n += __popc(bits);
            }
            const float top = warp_max(bg);
            const uint32_t who = __ballot_sync(full, bg == top);
            ba = __shfl_sync(full, ba, __ffs(who | 0x80000000u) - 1);
            if (lane == 0) {
                sh.nA = n;
                sh.top = n ? ba : 0u;
            }
        }
        __syncthreads();
        float maxaf = -INFINITY;   // largest G_f(a), a not in A+
        for (uint32_t ch = 0; ch < nch; ++ch) maxaf = fmaxf(maxaf, afch[ch]);
        // every template's shifts, a warp per template: chunk maxima, signs, rows (t, b)
        for (uint32_t t = warp; t < M; t += nwarps) {
            const float* gt = Gk + (uint64_t)t * S2;
            const float* lt = P.L + (uint64_t)t * d.N + p - S;   // lt[x], x in bounds, lies in the row
            const float room = (nx[t] + cst[t]) + maxaf;
            float gm = -INFINITY;
            for (uint32_t c0 = 0; c0 < nch; c0 += 8) {
                float g[8], lv[8];
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    const uint32_t x = (c0 + q) * 32 + lane;
                    const bool in = x >= xlo && x < xhi;   // false past the last chunk
                    g[q] = in ? gt[x] : -INFINITY;
                    lv[q] = in ? lt[x] : 0.f;
                }
                float mine = -INFINITY;
                uint32_t bits = 0;
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q) {
                    if (c0 + q >= nch) break;
                    const float m = warp_max(g[q]);
                    const uint32_t b = __ballot_sync(full, lv[q] > 0.f);
                    gm = fmaxf(gm, m);
                    if (lane == q) {
                        mine = m;
                        bits = b;
                    }
                    if (b == 0u) continue;
                    const uint32_t keep = __ballot_sync(full, lv[q] > 0.f && g[q] + room >= thr0);
                    if (keep == 0u) continue;
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&sh.nrows, (uint32_t)__popc(keep));
                    at = __shfl_sync(full, at, 0) + __popc(keep & below);
                    if (((keep >> lane) & 1u) && at < kRowCap) {
                        rowc[at] = (1u << 22) | (t << 10) | ((c0 + q) * 32 + lane);
                        rowg[at] = g[q];
                    }
                }
                if (lane < 8 && c0 + lane < nch) {
                    gch[(size_t)t * nch + c0 + lane] = mine;
                    pb[(size_t)t * nch + c0 + lane] = bits;
                }
            }
            if (lane == 0) gmax[t] = gm;
        }
        __syncthreads();
        // estimate of this lane's item in chunk ch of a row; -inf: no such item
        auto item = [&](uint32_t row, float g, uint32_t ch) -> float {
            const uint32_t y = row & 1023u, t = (row >> 10) & 4095u, x = ch * 32 + lane;
            const bool k1 = (row >> 22) != 0u;
            bool ok = x >= xlo && x < xhi && x + W >= y && x <= y + W;
            if (k1) ok = ok && !((pb[(size_t)f * nch + ch] >> lane) & 1u);
            const float v = !ok ? 0.f : (k1 ? Gf[x] : Gk[(uint64_t)t * S2 + x]);
            const float xv = ok && share[t] ? __ldg((k1 ? P.XTT : P.XT) + (((uint64_t)f * M + t) * S2 + y) * S2 + x) : 0.f;
            return ok ? (g + v) - xv : -INFINITY;
        };
        auto lower = [&]() { return fmaxf(__int_as_float(*(volatile int*)&sh.lb), thr0); };
        uint32_t nq = 0;   // chunks in this warp's queue
        // evaluates the queue's last (up to) eight chunks
        auto drain8 = [&]() {
            const uint32_t n = min(nq, 8u), b = nq - n;
            nq = b;
            evals += n;
            float v[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i)
                v[i] = i < n ? item(qc[b + i] & 0x7FFFFFu, qg[b + i], qc[b + i] >> 23) : -INFINITY;
            float m = -INFINITY;   // lane i < n: chunk i's largest estimate
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                const float w = warp_max(v[i]);
                if (lane == i) m = w;
            }
            const uint32_t code = lane < n ? qc[b + lane] : 0u;
            const float c = cst[(code >> 10) & 4095u];
            const float lb = warp_max(lane < n ? m - c : -INFINITY);
            if (lane == 0 && lb > __int_as_float(*(volatile int*)&sh.lb)) atomicMax(&sh.lb, __float_as_int(lb));
            if (lane < n && m + c >= fmaxf(lb, lower())) {
                const uint32_t at = atomicAdd(&sh.nchunks, 1u);
                if (at < kChunkCap) {
                    chc[at] = code;
                    chu[at] = m + c;
                    chg[at] = qg[b + lane];
                }
            }
            __syncwarp();
        };
        // Batches of 32 rows, one a lane: first the rows (a, t) of the largest G_f(a), over all
        // warps, then the other rows (a in A+, t), then the rows (t, b) with L_t(b) > 0, from
        // their list or, if they are more than it holds, word by word of the signs.  One
        // place in the code for all of them: copies of the evaluation overrun the
        // instruction cache (17 of 29 cycles per instruction waiting for it).
        const uint32_t nA = sh.nA, top = sh.top, nrow0 = nA * M, nrow1 = sh.nrows, ntask = M * nch;
        const bool listed = nrow1 <= kRowCap;
        const uint32_t n0 = (nrow0 + 31) / 32, n1 = listed ? (nrow1 + 31) / 32 : ntask;
#pragma unroll 1
        for (uint32_t phase = 0; phase < 2; ++phase) {
            const uint32_t last = phase ? n0 + n1 : (nA ? (M + 31) / 32 * nwarps : 0u);
#pragma unroll 1
            for (uint32_t i = warp; i < last; i += nwarps) {
                float ub = -INFINITY, g = 0.f;
                uint32_t row = 0;
                if (phase == 0 || i < n0) {
                    const uint32_t r = i * 32 + lane, ai = phase ? r / M : top;
                    const uint32_t t = phase ? r - ai * M : warp + nwarps * (lane + 32 * (i / nwarps));
                    if (phase ? (r < nrow0 && ai != top) : t < M) {
                        const uint32_t a = alist[ai];
                        g = Gf[a];
                        row = (t << 10) | a;
                        ub = ((g + gmax[t]) + nx[t]) + cst[t];
                    }
                } else if (listed) {
                    const uint32_t r = (i - n0) * 32 + lane;
                    if (r < nrow1) {
                        row = rowc[r];
                        g = rowg[r];
                        const uint32_t t = (row >> 10) & 4095u;
                        ub = ((g + maxaf) + nx[t]) + cst[t];
                    }
                } else {
                    const uint32_t e = i - n0, t = e / nch, x = (e - t * nch) * 32 + lane;
                    if ((pb[e] >> lane) & 1u) {
                        g = Gk[(uint64_t)t * S2 + x];
                        row = (1u << 22) | (t << 10) | x;
                        ub = ((g + maxaf) + nx[t]) + cst[t];
                    }
                }
                // the chunks that reach the lower bound, of the rows that do
                const float need = lower();
                const bool want = ub >= need;
                const uint32_t y = row & 1023u, t = (row >> 10) & 4095u;
                const bool k1 = (row >> 22) != 0u;
                const float* xc = k1 ? P.XCT + (((uint64_t)f * M + t) * S2 + y) * nch
                                     : P.XC + (((uint64_t)f * S2 + y) * M + t) * nch;
                const float* gm = k1 ? afch : gch + (size_t)t * nch;
                const bool sharing = want && share[t];
                const float gc = want ? g + cst[t] : -INFINITY;
                const uint32_t c1 = __any_sync(full, want) ? nch : 0u;
                const bool closing = i + nwarps >= last;   // this warp's last batch: empty the queue
                for (uint32_t c0 = 0; c0 < c1 || (closing && c0 == 0); c0 += 8) {
                    float xv[8];
                    uint32_t km = 0;
#pragma unroll
                    for (uint32_t q = 0; q < 8; ++q) xv[q] = sharing && c0 + q < nch ? __ldg(xc + c0 + q) : 0.f;
#pragma unroll
                    for (uint32_t q = 0; q < 8; ++q)
                        if (c0 + q < nch && (gm[c0 + q] + xv[q]) + gc >= need) km |= 1u << q;
                    uint32_t any = __reduce_or_sync(full, km);
                    const bool end = closing && c0 + 8 >= c1;
                    do {
                        if (any) {
                            const uint32_t q = __ffs(any) - 1;
                            any &= any - 1;
                            const bool mine = (km >> q) & 1u;
                            const uint32_t pm = __ballot_sync(full, mine), at = nq + __popc(pm & below);
                            if (mine) {
                                qc[at] = ((c0 + q) << 23) | row;
                                qg[at] = g;
                            }
                            nq += __popc(pm);
                            __syncwarp();
                        }
                        // evaluate while the queue has no room for 32 more, or at the end
                        while (nq > (end && any == 0u ? 0u : kQueue - 32u)) drain8();
                    } while (any);
                }
            }
            __syncthreads();
        }
        // the list of chunks too small for this window: look at every item instead
        const bool over = sh.nchunks > kChunkCap;
        const uint32_t nchunks = over ? 0u : sh.nchunks;
        // every item of the window, row by row: visit(row, chunk, estimates)
        auto every = [&](auto&& visit) {
            for (uint32_t r = warp; r < nA * M; r += nwarps) {
                const uint32_t ai = r / M, t = r - ai * M, a = alist[ai];
                for (uint32_t ch = 0; ch < nch; ++ch) visit((t << 10) | a, ch, item((t << 10) | a, Gf[a], ch));
            }
            for (uint32_t e = warp; e < ntask; e += nwarps) {
                const uint32_t t = e / nch;
                for (uint32_t bits = pb[e]; bits; bits &= bits - 1) {
                    const uint32_t b = (e - t * nch) * 32 + __ffs(bits) - 1, row = (1u << 22) | (t << 10) | b;
                    const float g = Gk[(uint64_t)t * S2 + b];
                    for (uint32_t ch = 0; ch < nch; ++ch) visit(row, ch, item(row, g, ch));
                }
            }
        };
        const float thr = fmaxf(__int_as_float(sh.lb), thr0);
        // list the items that reach it; where the global list is full, score them here
        unsigned long long kbest = 0ull;
        auto list_items = [&](uint32_t row, uint32_t ch, float est, bool here) {
            const uint32_t y = row & 1023u, t = (row >> 10) & 4095u, x = ch * 32 + lane;
            const bool k1 = (row >> 22) != 0u;
            const bool reach = est + cst[t] >= thr;
            const uint32_t m = __ballot_sync(full, reach);
            if (m == 0u) return;
            const uint32_t a = k1 ? x : y, b = k1 ? y : x;
            if (!here) {
                uint32_t base = 0;
                if (lane == 0) base = atomicAdd(&P.status->cand_count, (uint32_t)__popc(m));
                const uint32_t at = __shfl_sync(full, base, 0) + __popc(m & ((1u << lane) - 1u));
                if (!reach) return;
                if (at < P.cand_cap)
                    P.gcand[at] = ((unsigned long long)kk << 32) | ((unsigned long long)t << 20) |
                                  ((unsigned long long)a << 10) | (unsigned long long)b;
                else
                    sh.full = 1;
                return;
            }
            if (!reach) return;
            const float v = pair_exact_call(d, P.T, P.V, f, t, p, a, b, P.chmask[f] | P.chmask[t]);
            if (!(v > 0.f)) return;
            const uint64_t r0 = (uint64_t)t + (uint64_t)M * a + (uint64_t)M * S2 * b;
            uint32_t pr = item_priority(r0, d.WG, lbits);
            for (uint64_t rr = r0 + items; rr < slots; rr += items) pr = min(pr, item_priority(rr, d.WG, lbits));
            const unsigned long long key =
                ((unsigned long long)__float_as_uint(v) << 32) | (unsigned long long)(0xFFFFFFFFu - pr);
            kbest = key > kbest ? key : kbest;
        };
        auto list_window = [&](bool here) {
            if (over) {
                every([&](uint32_t row, uint32_t ch, float est) {
                    list_items(row, ch, est, here);
                    __syncwarp();
                });
                return;
            }
            for (uint32_t e = warp; e < nchunks; e += nwarps) {
                if (!(chu[e] >= thr)) continue;
                const uint32_t row = chc[e] & 0x7FFFFFu, ch = chc[e] >> 23;
                list_items(row, ch, item(row, chg[e], ch), here);
                __syncwarp();
            }
        };
#pragma unroll 1
        for (int here = 0; here < 2; ++here) {
            list_window(here != 0);
            __syncthreads();
            if (!sh.full) break;   // the same for the whole CTA
            if (!here) continue;
            if (kbest) atomicMax(&sh.best, kbest);
            __syncthreads();
            if (threadIdx.x == 0 && sh.best) atomicMax(&P.keys[P.k0 + kk], sh.best);
        }
    }
    if (lane == 0 && evals) atomicAdd(&P.status->pair_items, 32ull * evals);
}

// Screening order of a batch of flagged windows: grouped by best label f (a
// counting sort), so CTAs running at the same time read the same template's
// cross-term slices from L2.  Windows past the flagged count go last.
__global__ void __launch_bounds__(1024) label_order_kernel(Dims d, const uint32_t* __restrict__ flag,
                                                           const DevStatus* status,
                                                           const uint32_t* __restrict__ best_lab, uint32_t k0,
                                                           uint32_t kc, uint32_t* order)
{
    extern __shared__ uint32_t hist[];   // [M + 1]
    const uint32_t nflag = flagged_windows(status), M = d.M;
    for (uint32_t i = threadIdx.x; i <= M; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < kc; j += blockDim.x) {
        const uint32_t f = k0 + j < nflag ? min(best_lab[flag[k0 + j]], M) : M;
        atomicAdd(&hist[f], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (uint32_t i = 0; i <= M; ++i) { const uint32_t c = hist[i]; hist[i] = run; run += c; }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < kc; j += blockDim.x) {
        const uint32_t f = k0 + j < nflag ? min(best_lab[flag[k0 + j]], M) : M;
        order[atomicAdd(&hist[f], 1u)] = j;
    }
}

// Exact scores of the listed candidates, entry = window slot kk (32 bits) | t (12) |
// a (10) | b (10), in the reference's float order (pair_exact_g).  Folds the
// canonical winner key into keys[k0 + kk].
//
// A warp takes up to 16 candidates.  Channel by channel of each candidate's own
// non-zero ones, 32 taps at a time, the lanes form the products of one candidate
// after the other (a product rounds the same wherever it is formed) in shared memory;
// then lane e adds candidate e's products with the window and lane 16 + e its squares,
// one by one in tap order.  The loads of eight candidates are in flight together,
// where a thread per candidate waited for its own at every eighth tap: per pursuit
// 16.8 -> 2.7 ms (20 s of 64 channels x 200 templates, 0.16 M candidates in 36
// launches), 1.04 -> 0.39 ms (43 s of 11 x 27), 0.20 -> 0.17 ms (30 s of 4 x 6); with
// 1.2 M candidates (300 s of 16 x 40) the two are alike, 3.6 and 3.8 ms.  Fewer
// candidates a warp when there are not enough to fill the SMs.
constexpr int kScoreThreads = 128;
constexpr uint32_t kScoreMany = 16;

__global__ void __launch_bounds__(kScoreThreads) score_kernel(
    Dims d, const float* __restrict__ V, const float* __restrict__ T, const uint32_t* __restrict__ flag, uint32_t k0,
    const uint32_t* __restrict__ best_lab, const uint32_t* __restrict__ best_idx,
    const unsigned long long* __restrict__ gcand, uint32_t cap, DevStatus* status, unsigned long long* keys,
    const unsigned long long* __restrict__ chmask)
{
    __shared__ float prod[kScoreThreads / 32][2 * kScoreMany * 33];   // [kind][candidate][32 taps, padded]
    __shared__ uint4 rows[kScoreThreads / 32][kScoreMany];            // template rows and voltage row of the channel
    __shared__ int2 shift[kScoreThreads / 32][kScoreMany];            // first template samples
    const uint32_t n = min(status->cand_count, cap);
    const uint32_t S2 = 2 * d.S + 1, M = d.M, C = d.C, W = d.W;
    const uint64_t items = (uint64_t)S2 * S2 * M;
    const uint64_t slots = ((items - 1) / d.WG + 1) * d.WG;
    uint32_t lbits = 0;
    while ((1u << lbits) < d.WG) ++lbits;
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, e = lane & 15u;
    const uint32_t nwarps = gridDim.x * (kScoreThreads / 32);
    uint32_t G = kScoreMany;
    while (G > 2 && (n + G - 1) / G < nwarps) G >>= 1;
    float* mine = prod[warp] + (lane >> 4) * (kScoreMany * 33) + e * 33;
    for (uint32_t i0 = (blockIdx.x * (kScoreThreads / 32) + warp) * G; i0 < n; i0 += nwarps * G) {
        // candidate e on lanes e and 16 + e
        const uint32_t have = min(G, n - i0);
        const unsigned long long code = e < have ? gcand[i0 + e] : ~0ull;
        const uint32_t kk = (uint32_t)(code >> 32);
        const uint32_t t = (uint32_t)(code >> 20) & 0xFFFu, a = (uint32_t)(code >> 10) & 0x3FFu, b = (uint32_t)code & 0x3FFu;
        const bool ok = code != ~0ull && (uint64_t)k0 + kk < flagged_windows(status) && t < M && a < S2 && b < S2;
        uint32_t f = 0, p = 0;
        unsigned long long left = 0ull;   // channels still to sum (C <= 64)
        if (ok) {
            const uint32_t id = flag[k0 + kk];
            f = best_lab[id];
            p = best_idx[id];
            left = chmask[f] | chmask[t];
        }
        uint32_t next = 0;                // channel (C > 64: all of them)
        if (lane < kScoreMany) shift[warp][e] = make_int2((int)d.S - (int)a, (int)d.S - (int)b);
        // blocks of 32 taps of a channel, eight candidates at a time
        bool on = false;                  // this candidate takes part in the channel
        uint32_t act = 0, j0 = W, g0 = 0;
        auto advance = [&]() {            // to the next eight, block or channel; act == 0: done
            g0 += 8;
            if (g0 < G && ((act >> g0) & 0xFFu)) return;
            g0 = 0;
            j0 += 32;
            if (j0 < W) return;
            on = ok && (C > 64 ? next < C : left != 0ull);
            act = __ballot_sync(full, on) & 0xFFFFu;
            const uint32_t c = C > 64 ? next : (uint32_t)__ffsll((long long)left) - 1u;
            if (on) {
                left &= left - 1;
                ++next;
                if (lane < kScoreMany) {
                    const uint64_t vo = (uint64_t)c * d.N + p;
                    rows[warp][e] = make_uint4((f * C + c) * W, (t * C + c) * W, (uint32_t)vo, (uint32_t)(vo >> 32));
                }
            }
            __syncwarp();
            j0 = 0;
        };
        float fv[8], tv[8], vv[8];
        auto fetch = [&]() {
            const uint32_t j = j0 + lane;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
                fv[q] = tv[q] = vv[q] = 0.f;
                if (!((act >> (g0 + q)) & 1u)) continue;   // the same for the whole warp
                const uint4 r = rows[warp][g0 + q];
                const int2 s = shift[warp][g0 + q];
                const int jf = (int)j + s.x, jt = (int)j + s.y;
                if (j < W) {
                    vv[q] = __ldg(V + (((uint64_t)r.w << 32) | r.z) + j);
                    if (jf >= 0 && jf < (int)W) fv[q] = __ldg(T + r.x + jf);
                    if (jt >= 0 && jt < (int)W) tv[q] = __ldg(T + r.y + jt);
                }
            }
        };
        float acc = 0.f, sum = 0.f;       // acc: lanes < 16
        advance();
        fetch();
        while (act) {
            const uint32_t cact = act, cj0 = j0, cg0 = g0;
            const bool con = on, last = cg0 + 8 >= G || ((cact >> (cg0 + 8)) & 0xFFu) == 0u;
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q) {
                if (!((cact >> (cg0 + q)) & 1u)) continue;
                const float sv = fadd(fv[q], tv[q]);
                prod[warp][(cg0 + q) * 33 + lane] = fmul(sv, vv[q]);
                prod[warp][(kScoreMany + cg0 + q) * 33 + lane] = fmul(sv, sv);
            }
            __syncwarp();
            advance();
            fetch();   // on its way during the sums
            if (!last) continue;
            if (cj0 == 0) sum = lane < kScoreMany ? acc : 0.f;
            if (con) {
                const uint32_t m = min(32u, W - cj0);
                if (m == 32u) {
#pragma unroll
                    for (uint32_t k = 0; k < 32; ++k) sum = fadd(sum, mine[k]);
                } else {
#pragma unroll 4
                    for (uint32_t k = 0; k < m; ++k) sum = fadd(sum, mine[k]);
                }
            }
            if (cj0 + 32 >= W) {
                const float ss = __shfl_sync(full, sum, lane | 16u);
                if (con && lane < kScoreMany) acc = ss > 0.f ? fsub(sum, fmul(0.5f, ss)) : sum;
            }
            __syncwarp();
        }
        if (ok && lane < kScoreMany && acc > 0.f) {
            const uint64_t r = (uint64_t)t + (uint64_t)M * a + (uint64_t)M * S2 * b;
            uint32_t pr = item_priority(r, d.WG, lbits);
            for (uint64_t rr = r + items; rr < slots; rr += items) pr = min(pr, item_priority(rr, d.WG, lbits));
            atomicMax(&keys[k0 + kk],
                      ((unsigned long long)__float_as_uint(acc) << 32) | (unsigned long long)(0xFFFFFFFFu - pr));
        }
        const uint32_t done = __popc(__ballot_sync(full, ok) & 0xFFFFu);
        if (lane == 0 && done) atomicAdd(&status->n_pair_exact, done);
    }
}

}  // namespace

// Whether a call's partial correlations are made by transforms: wherever they
// apply (W + S <= 256 and the channels' spectra fit shared memory), unless the
// caller asked for a template group of the direct kernel.  Measured against it,
// per pursuit: 16 channels x 40 templates, 300 s 31.8 -> 6.0 ms; 64 x 200, 20 s
// 38.8 -> 11.3 ms; 11 x 27 without zero channels, 43 s 2.3 -> 0.8 ms; 4 x 5, 5 s
// 0.16 -> 0.08 ms.
static bool window_corr_by_fft(const Dims& d) { return fft_windows_supported(d) && tuning().pc_group == 0; }

struct PcConfig {
    int Q = 0;
    size_t smem = 0;
};

// The partial-correlation launch shape of the calling thread's current chunk:
// launch_overlap_tables sets it and launch_overlap_fast reads it, both inside the
// same fbp_pursue_chunk call on that thread, so no other call can come between them.
PcConfig& pc_config()
{
    static thread_local PcConfig c;
    return c;
}

int launch_overlap_tables(const Dims& d, const Work& w, const float* T, cudaStream_t st)
{
    const Layout& L = *w.lay;
    if (!L.screened) return FBP_OK;
    const unsigned long long* chmask = w.at<unsigned long long>(L.off_tchm);
    float* mx = w.at<float>(L.off_mx);
    count_launch(2);
    energy_table_kernel<<<d.M, 128, (d.W + 1) * 8, st>>>(d, T, w.at<float2>(L.off_et), mx + (size_t)d.M * d.M);
    auto cross_smem = [&](int lags) { return (size_t)2 * d.C * d.W * 4 + (size_t)lags * ((d.W + 1) | 1u) * 8; };
    const int lags = cross_smem(32) <= 100 * 1024 ? 32 : 16;   // two CTAs per SM, or the shorter chunk
    if (cross_smem(lags) > 201 * 1024) return fail(FBP_E_ARG, "template too large for the pair table kernel");
    FBP_CUDA(allow_max_dyn_smem(cross_table_kernel));
    const uint32_t pairs = d.M * d.M, groups = (2 * std::min(d.W, 2 * d.S) + lags) / lags;
    const uint32_t split = std::max(1u, std::min(groups, 148u * 2 / pairs));
    cross_table_kernel<<<dim3(pairs, split), kCrossThreads, cross_smem(lags), st>>>(
        d, T, chmask, lags, w.at<float>(L.off_xt), w.at<float>(L.off_xtt), w.at<float>(L.off_xc), w.at<float>(L.off_xct),
        mx);
    if (split > 1) {
        count_launch();
        cross_bound_kernel<<<dim3(pairs, (2 * d.S + 8) / 8), kCrossThreads, 0, st>>>(   // two rows a warp
            d, chmask, w.at<float>(L.off_xt), w.at<float>(L.off_xtt), w.at<float>(L.off_xc), w.at<float>(L.off_xct), mx);
    }
    FBP_CUDA(cudaGetLastError());
    if (window_corr_by_fft(d)) return FBP_OK;
    count_launch();
    template_order_kernel<<<1, 256, d.M * 4, st>>>(d, w.at<uint8_t>(L.off_clist), w.at<uint32_t>(L.off_ccnt),
                                                  w.at<uint32_t>(L.off_perm));
    FBP_CUDA(cudaGetLastError());
    // channel unions of the template groups decide how many templates a direct
    // partial-correlation CTA can stage: read the order and masks back once
    std::vector<uint32_t> perm(d.M);
    std::vector<unsigned long long> mask(d.M);
    FBP_CUDA(cudaMemcpyAsync(perm.data(), w.at<uint32_t>(L.off_perm), d.M * 4, cudaMemcpyDeviceToHost, st));
    FBP_CUDA(cudaMemcpyAsync(mask.data(), chmask, d.M * 8, cudaMemcpyDeviceToHost, st));
    FBP_CUDA(cudaStreamSynchronize(st));
    PcConfig& pc = pc_config();
    pc.Q = 0;
    // group size: least estimated work, sum over groups of Q x (union channels),
    // weighted by the measured cost per multiply-add of each group size (two
    // strip loads feed Q templates; below 4 the shared-memory loads dominate)
    double best = 0.0;
    const int want_q = (int)tuning().pc_group;
    for (int Q = 8; Q >= 1; Q >>= 1) {
        if (want_q && Q > want_q) continue;
        // measured time per unit of work relative to Q = 4: Q = 8 0.72 (64 ch, 200
        // templates, 60 s) and 0.84 (16 ch, 40 templates, 10 min), Q = 2 1.0-1.2, Q = 1 1.3-1.4
        const double eff = Q >= 8 ? 0.78 : (Q == 4 ? 1.0 : (Q == 2 ? 1.2 : 1.6));
        uint32_t cu_max = 0;
        double work = 0.0;
        for (uint32_t g0 = 0; g0 < d.M; g0 += Q) {
            unsigned long long m = 0ull;
            for (uint32_t q = 0; q < (uint32_t)Q && g0 + q < d.M; ++q) m |= mask[perm[g0 + q]];
            uint32_t cu = 0;
            for (uint32_t c = 0; c < d.C; ++c) cu += (c >= 64 || ((m >> c) & 1ull)) ? 1u : 0u;
            cu_max = cu > cu_max ? cu : cu_max;
            work += (double)Q * cu;
        }
        const size_t smem = pc_smem_bytes(d, cu_max, Q);
        if (!(smem <= 110 * 1024 || (Q == 1 && smem <= 200 * 1024))) continue;
        if (want_q) {   // the caller's group size, or the largest feasible one below it
            pc.Q = Q;
            pc.smem = smem;
            break;
        }
        if (pc.Q == 0 || work * eff < best) {
            pc.Q = Q;
            pc.smem = smem;
            best = work * eff;
        }
    }
    return FBP_OK;
}

int launch_overlap_fast(const Dims& d, const Work& w, const float* V, const float* T, const float* theta,
                        uint32_t nflag_max, cudaStream_t st)
{
    const Layout& L = *w.lay;
    if (!L.screened) return launch_overlap_plain(d, w, V, T, theta, nflag_max, st);
    if (nflag_max == 0) return FBP_OK;
    const uint32_t S2 = 2 * d.S + 1;
    if (S2 > 1024 || d.C > 256 || d.M > 4096) return launch_overlap_plain(d, w, V, T, theta, nflag_max, st);
    const PcConfig pc = pc_config();
    const int Q = pc.Q;
    const size_t smem_a = pc.smem;
    const bool fft = window_corr_by_fft(d);
    if (Q == 0 && !fft) return launch_overlap_plain(d, w, V, T, theta, nflag_max, st);
    const uint32_t pc_threads = 32u * std::min<uint32_t>((S2 + 15) / 16, kPcMaxWarps);
    if (screen_smem_bytes(d.M, S2, d.C, kScrThreads) > 200 * 1024)
        return launch_overlap_plain(d, w, V, T, theta, nflag_max, st);
    const bool wide = nflag_max <= kScrFewWindows && screen_smem_bytes(d.M, S2, d.C, kScrWideThreads) <= 100 * 1024;
    const int scr_threads = wide ? kScrWideThreads : kScrThreads;
    const size_t smem_b = screen_smem_bytes(d.M, S2, d.C, scr_threads);
    const auto screen = wide ? screen_kernel<kScrWideThreads, kScrWidePerSm> : screen_kernel<kScrThreads, kScrPerSm>;
    FBP_CUDA(allow_max_dyn_smem(screen));
    int scr_per_sm = 1;
    FBP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&scr_per_sm, screen, scr_threads, smem_b));
    const uint32_t groups = Q > 0 ? (d.M + Q - 1) / Q : 0u;
    float* G = w.at<float>(L.off_g);
    const float2* Et = w.at<float2>(L.off_et);
    const uint32_t* perm = w.at<uint32_t>(L.off_perm);
    const unsigned long long* chm = w.at<unsigned long long>(L.off_tchm);
    ScreenArgs P;
    P.d = d;
    P.V = V;
    P.T = T;
    P.L = w.L();
    P.theta = theta;
    P.XT = w.at<float>(L.off_xt);
    P.XTT = w.at<float>(L.off_xtt);
    P.XC = w.at<float>(L.off_xc);
    P.XCT = w.at<float>(L.off_xct);
    P.mx = w.at<float>(L.off_mx);
    P.G = G;
    P.vc2 = fft ? w.at<float>(L.off_vc2) : nullptr;
    P.z2 = fft ? w.at<float>(L.off_z2) : nullptr;
    P.flag = w.flag();
    P.status = w.status();
    P.best_lab = w.best_lab();
    P.best_idx = w.best_idx();
    P.best_lik = w.best_lik();
    P.keys = w.keys();
    P.gcand = w.at<unsigned long long>(L.off_cand);
    P.cand_cap = (uint32_t)L.cand_cap;
    P.chmask = chm;
    P.order = w.at<uint32_t>(L.off_order);
    for (uint32_t k0 = 0; k0 < nflag_max; k0 += (uint32_t)L.gbatch) {
        const uint32_t kc = (uint32_t)((nflag_max - k0) < L.gbatch ? (nflag_max - k0) : L.gbatch);
        count_launch(2);
        if (fft) {
        KScope ks(&fbp_chunk_stats::ms_partial_corr, st);
        FBP_TRY(launch_window_corr(d, w, V, theta, Et, k0, kc, G, w.at<float>(L.off_vc2), w.at<float>(L.off_z2), st));
        } else {
        KScope ks(&fbp_chunk_stats::ms_partial_corr, st);
        count_launch();
        // persistent over the windows: as many CTAs as fit resident, split over the template groups
#define FBP_PC(QQ)                                                                                            \
    case QQ: {                                                                                                \
        FBP_CUDA(allow_max_dyn_smem(partial_corr_kernel<QQ>));                                                          \
        int per_sm = 1;                                                                                       \
        FBP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, partial_corr_kernel<QQ>,              \
                                                               (int)pc_threads, smem_a));                 \
        const uint32_t want = (uint32_t)((148u * (per_sm > 0 ? per_sm : 1) + groups - 1) / groups);           \
        const uint32_t slices = std::min<uint32_t>((kc + kPcWin - 1) / kPcWin, want);                         \
        partial_corr_kernel<QQ><<<dim3(slices, groups), pc_threads, smem_a, st>>>(                          \
            d, V, T, w.L(), theta, Et, perm, chm, w.flag(), w.status(), w.best_lab(), w.best_idx(), k0, kc, G); \
        break;                                                                                                \
    }
        switch (Q) {
            FBP_PC(8)
            FBP_PC(4)
            FBP_PC(2)
            FBP_PC(1)
        }
#undef FBP_PC
        }
        uint32_t* order = w.at<uint32_t>(L.off_order);
        count_launch();
        label_order_kernel<<<1, 1024, (d.M + 1) * 4, st>>>(d, w.flag(), w.status(), w.best_lab(), k0, kc, order);
        if (k0 > 0) FBP_CUDA(cudaMemsetAsync(&w.status()->cand_count, 0, 4, st));   // the pass starts with 0
        {
        KScope ks(&fbp_chunk_stats::ms_screen, st);
        P.k0 = k0;
        P.kc = kc;
        const uint32_t grid = std::min<uint32_t>(kc, 148u * (scr_per_sm > 0 ? scr_per_sm : 1));
        screen<<<grid, scr_threads, smem_b, st>>>(P);
        }
        KScope ks(&fbp_chunk_stats::ms_score, st);
        score_kernel<<<148 * 6, kScoreThreads, 0, st>>>(d, V, T, w.flag(), k0, w.best_lab(), w.best_idx(), P.gcand,
                                              (uint32_t)L.cand_cap, w.status(), w.keys(), chm);
        FBP_CUDA(cudaGetLastError());
    }
    return FBP_OK;
}

}  // namespace fbp
