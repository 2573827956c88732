// adjoint.cu -- residual energy of a fixed spike assignment and its gradient.
//
// Template refinement at fixed assignments (no counterpart in the reference):
//     r(c, x) = v(c, x) - sum_k a_k * T~_k(c, x - s_k)
//     E       = sum_{c,x} r(c, x)^2
// where spike k has onset s_k (the pursuit's event index), label l_k, amplitude
// a_k and fractional shift tau_k in (-1, 1) samples, and T~ is template l_k moved
// right by tau_k with linear interpolation:
//     u = |tau|, dir = tau >= 0 ? -1 : +1
//     T~(c, j) = (1 - u) T(c, j) + u T(c, j + dir),   j in [-1, W]   (T = 0 outside [0, W))
// Samples outside [0, N) are not modelled.  Gradients:
//     dE/da_k     = -2 sum_{c,j} T~_k(c, j) r(c, s_k + j)
//     dE/dtau_k   = -2 a_k sgn(tau_k) sum_{c,j} (T(c, j + dir) - T(c, j)) r(c, s_k + j)
//                   (sgn(0) = +1: the tau >= 0 branch)
//     dE/dT_l(c,i)= -2 sum_{k: l_k = l} a_k ((1 - u) r(c, s_k + i) + u r(c, s_k + i - dir))
// Nothing is stored between the loss and the gradient: residual values are rebuilt in
// FP64 registers from the voltage and every spike whose support meets them (spikes
// sorted by onset).  A warp takes 128 samples of one channel, four a lane, and the
// spikes one after the other in onset order; a template row that is zero there is
// left out (its product is exactly 0; not when amplitude or shift is not finite).
// Sums run in FP64; template gradients accumulate with FP64 atomics.
//
// Bound by instruction issue: one CTA a spike over a (channel, sample) index with a
// division and 64-bit compares an element took 469 us for the loss (and 122 us more
// for the sum of v^2) and 521 us for the gradient at 16 channels x 60 s, 19200 spikes of
// 101 samples, with the FP64 pipe 6-9% and the L2's atomics 9% busy; as here: 137 us and
// 242 us.
#include <algorithm>

#include <cub/cub.cuh>

#include "fbp_internal.cuh"

namespace fbp {
namespace {

constexpr int kAdjThreads = 128;

struct AdjArgs {
    uint32_t C, N, M, W;
    const float* V;        // [C][N]
    const float* T;        // [M][C][W]
    const uint32_t* idx;   // [n] onsets, ascending
    const uint32_t* lab;   // [n]
    const float* amp;      // [n]
    const float* tau;      // [n]
    uint32_t n;
};

constexpr int kAdjWarps = kAdjThreads / 32;
constexpr int kAdjCols = 4;                 // columns a lane
constexpr int kAdjSpan = 32 * kAdjCols;     // columns a warp

// One spike as a warp's rows meet it
struct AdjSpike {
    double a, u;      // amplitude, |shift|
    int32_t off;      // column of the template's sample 0
    int32_t dir;      // -1 or +1
    uint32_t lab;
    uint32_t finite;  // amplitude and shift are finite
};

__device__ __forceinline__ AdjSpike adj_spike(const AdjArgs& A, uint32_t k, int64_t x0)
{
    AdjSpike s;
    const double t = A.tau[k];
    s.a = A.amp[k];
    s.u = t >= 0.0 ? t : -t;
    s.dir = t >= 0.0 ? -1 : 1;
    s.off = (int32_t)((int64_t)A.idx[k] - x0);
    s.lab = A.lab[k];
    s.finite = isfinite(s.a) && isfinite(s.u);
    return s;
}

// first spike with onset >= key (a warp, 32 probes a step)
__device__ uint32_t first_onset(const AdjArgs& A, int64_t key)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = A.n;   // below lo: onset < key; from hi on: >= key
    while (lo < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t at = (uint64_t)lo + (uint64_t)lane * step;
        const bool less = at < hi && (int64_t)A.idx[at] < key;
        const uint32_t c = __popc(__ballot_sync(0xffffffffu, less));   // probes 0 .. c-1 are below
        if (c == 0) return lo;
        const uint64_t top = (uint64_t)lo + (uint64_t)c * step;
        lo = lo + (c - 1) * step + 1;
        hi = top < hi ? (uint32_t)top : hi;
    }
    return lo;
}

// r[i] = residual of channel c at sample x0 + lane + 32 i (0 outside [0, N)), from
// the spikes [k0, k1); `box` is the warp's, and holds those spikes already if `held`.
__device__ __forceinline__ void residual_row(const AdjArgs& A, uint32_t c, int64_t x0, uint32_t k0, uint32_t k1,
                                             AdjSpike* box, bool held, double (&r)[kAdjCols])
{
    const int lane = threadIdx.x & 31;
    const float* v = A.V + ((int64_t)((uint64_t)c * A.N) + x0 + lane);
    // columns [first, last) are samples of the recording
    const int first = x0 < 0 ? (int)-x0 : 0;
    const int last = x0 + kAdjSpan <= (int64_t)A.N ? kAdjSpan : (int)max((int64_t)A.N - x0, (int64_t)0);
#pragma unroll
    for (int i = 0; i < kAdjCols; ++i) {
        const int q = lane + 32 * i;
        r[i] = q >= first && q < last ? (double)v[32 * i] : 0.0;
    }
    for (uint32_t kb = k0; kb < k1; kb += 32) {
        const uint32_t m = min(32u, k1 - kb);
        if (!held) {
            __syncwarp();
            if (lane < (int)m) box[lane] = adj_spike(A, kb + lane, x0);
            __syncwarp();
        }
        for (uint32_t i0 = 0; i0 < m; ++i0) {
            const AdjSpike s = box[i0];
            if (s.lab >= A.M) continue;
            const float* Tc = A.T + ((uint64_t)s.lab * A.C + c) * A.W;
            float ta[kAdjCols], tb[kAdjCols];   // zero outside the support
            bool some = !s.finite;
            const int j0 = lane - s.off;
            const float *pa = Tc + j0, *pb = pa + s.dir;
#pragma unroll
            for (int i = 0; i < kAdjCols; ++i) {
                const int j = j0 + 32 * i;
                ta[i] = (uint32_t)j < A.W ? pa[32 * i] : 0.f;
                tb[i] = (uint32_t)(j + s.dir) < A.W ? pb[32 * i] : 0.f;
                some |= ta[i] != 0.f || tb[i] != 0.f;
            }
            if (!__any_sync(0xffffffffu, some)) continue;
#pragma unroll
            for (int i = 0; i < kAdjCols; ++i)
                if (s.finite || (uint32_t)(j0 + 32 * i + 1) < A.W + 2)
                    r[i] -= s.a * ((1.0 - s.u) * (double)ta[i] + s.u * (double)tb[i]);
        }
    }
    if (first > 0 || last < kAdjSpan) {
#pragma unroll
        for (int i = 0; i < kAdjCols; ++i) {
            const int q = lane + 32 * i;
            if (q < first || q >= last) r[i] = 0.0;
        }
    }
}

// E: a warp takes 128 samples of every slices-th channel at a time: of all channels where
// the recording has samples enough to fill the SMs, else of a share of them (64 channels x
// 100,000 samples, 300 spikes, 89 us by all channels a warp, now 24).
template <bool SLICED>
__global__ void __launch_bounds__(kAdjThreads) adjoint_loss_kernel(AdjArgs A, uint32_t slices, double* loss)
{
    typedef cub::BlockReduce<double, kAdjThreads> R;
    __shared__ typename R::TempStorage tmp;
    __shared__ AdjSpike box[kAdjWarps][32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t nseg = ((uint64_t)A.N + kAdjSpan - 1) / kAdjSpan;
    if (!SLICED) slices = 1;
    double acc = 0.0;
    for (uint64_t g = (uint64_t)blockIdx.x * kAdjWarps + warp; g < nseg * slices; g += (uint64_t)gridDim.x * kAdjWarps) {
        const uint64_t seg = SLICED ? g / slices : g;
        const int64_t x0 = (int64_t)(seg * kAdjSpan);
        const uint32_t k0 = first_onset(A, x0 - (int64_t)A.W);
        uint32_t k1 = k0;   // past the last spike with onset <= x0 + 128
        for (;;) {
            const bool meets = (uint64_t)k1 + lane < A.n && (int64_t)A.idx[k1 + lane] <= x0 + kAdjSpan;
            const uint32_t ones = __popc(__ballot_sync(0xffffffffu, meets));
            k1 += ones;
            if (ones < 32) break;
        }
        const bool one = k1 - k0 <= 32;
        if (one) {
            __syncwarp();
            if (lane < k1 - k0) box[warp][lane] = adj_spike(A, k0 + lane, x0);
            __syncwarp();
        }
        for (uint32_t c = (uint32_t)(g - seg * slices); c < A.C; c += slices) {
            double r[kAdjCols];
            residual_row(A, c, x0, k0, k1, box[warp], one, r);
#pragma unroll
            for (int i = 0; i < kAdjCols; ++i) acc += r[i] * r[i];
        }
    }
    const double s = R(tmp).Sum(acc);
    if (threadIdx.x == 0) atomicAdd(loss, s);
}

// A CTA takes a spike, a warp every WARPS-th channel; a row's W + 2 columns are taken 126
// at a time, with one more on either side for the shifted residual.  Four warps, or 16
// where few spikes of many channels leave the SMs idle (300 spikes of 64 channels x 20
// samples 45 us, now 29; 60 of 128 x 76 85 us, now 33).
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 32 / WARPS) adjoint_grad_kernel(AdjArgs A, double scale, double* gT,
                                                                              float* g_amp, float* g_tau)
{
    __shared__ AdjSpike box[WARPS][32];
    __shared__ double part[2][WARPS];
    const int W = (int)A.W, TL = W + 2;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t k = blockIdx.x; k < A.n; k += gridDim.x) {
        const int64_t s = A.idx[k];
        const uint32_t l = A.lab[k];
        double da = 0.0, dt = 0.0;
        if (l < A.M) {
            const AdjSpike own = adj_spike(A, k, 0);
            uint32_t k0 = k, k1 = k + 1;   // the spikes whose support meets [s - 1, s + W]
            for (;;) {
                const bool meets = k0 > lane && (int64_t)A.idx[k0 - 1 - lane] >= s - W - 1;
                const uint32_t ones = __popc(__ballot_sync(0xffffffffu, meets));
                k0 -= ones;
                if (ones < 32) break;
            }
            for (;;) {
                const bool meets = (uint64_t)k1 + lane < A.n && (int64_t)A.idx[k1 + lane] <= s + W + 1;
                const uint32_t ones = __popc(__ballot_sync(0xffffffffu, meets));
                k1 += ones;
                if (ones < 32) break;
            }
            for (int q0 = 0; q0 < TL; q0 += kAdjSpan - 2) {
                const int64_t x0 = s - 2 + q0;   // column 0 of the row; its column p is the tile's q0 - 1 + p
                const bool one = k1 - k0 <= 32;
                if (one) {
                    __syncwarp();
                    if (lane < k1 - k0) box[warp][lane] = adj_spike(A, k0 + lane, x0);
                    __syncwarp();
                }
                for (uint32_t c = warp; c < A.C; c += WARPS) {
                    double r[kAdjCols];
                    residual_row(A, c, x0, k0, k1, box[warp], one, r);
                    const int j0 = q0 + (int)lane - 2;   // template sample of column `lane`
                    const float* pa = A.T + ((uint64_t)l * A.C + c) * A.W + j0;
                    const float* pb = pa + own.dir;
                    double* gc = gT + ((uint64_t)l * A.C + c) * A.W + j0;
                    float ta[kAdjCols], tb[kAdjCols];
                    bool some = false;
                    double next[kAdjCols];   // the column at q - dir
#pragma unroll
                    for (int i = 0; i < kAdjCols; ++i) {
                        const int j = j0 + 32 * i;
                        ta[i] = (uint32_t)j < A.W ? pa[32 * i] : 0.f;
                        tb[i] = (uint32_t)(j + own.dir) < A.W ? pb[32 * i] : 0.f;
                        some |= ta[i] != 0.f || tb[i] != 0.f || !isfinite(r[i]);
                        next[i] = __shfl_sync(0xffffffffu, r[i], (lane - own.dir) & 31);
                    }
                    if (own.dir < 0) {
#pragma unroll
                        for (int i = 0; i < kAdjCols; ++i)
                            if (lane == 31) next[i] = i + 1 < kAdjCols ? next[i + 1 < kAdjCols ? i + 1 : i] : 0.0;
                    } else {
#pragma unroll
                        for (int i = kAdjCols - 1; i >= 0; --i)
                            if (lane == 0) next[i] = i > 0 ? next[i > 0 ? i - 1 : 0] : 0.0;
                    }
                    if (__any_sync(0xffffffffu, some)) {
#pragma unroll
                        for (int i = 0; i < kAdjCols; ++i) {
                            const int p = lane + 32 * i;
                            if (p < 1 || p > kAdjSpan - 2 || j0 + 32 * i > W) continue;
                            da += ((1.0 - own.u) * (double)ta[i] + own.u * (double)tb[i]) * r[i];
                            dt += ((double)tb[i] - (double)ta[i]) * r[i];
                        }
                    }
                    // template sample j: (1 - u) r(s + j) + u r(s + j - dir)
#pragma unroll
                    for (int i = 0; i < kAdjCols; ++i) {
                        const int p = lane + 32 * i;
                        if (p >= 1 && p <= kAdjSpan - 2 && (uint32_t)(j0 + 32 * i) < A.W)
                            atomicAdd(&gc[32 * i], -2.0 * scale * own.a * ((1.0 - own.u) * r[i] + own.u * next[i]));
                    }
                }
            }
            dt *= -own.dir * own.a;   // sgn(tau) = -dir
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            da += __shfl_down_sync(0xffffffffu, da, o);
            dt += __shfl_down_sync(0xffffffffu, dt, o);
        }
        __syncthreads();   // the previous spike's sums have been read
        if (lane == 0) {
            part[0][warp] = da;
            part[1][warp] = dt;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            double sa = 0.0, st = 0.0;
            for (int w = 0; w < WARPS; ++w) {
                sa += part[0][w];
                st += part[1][w];
            }
            g_amp[k] = (float)(-2.0 * scale * sa);
            g_tau[k] = (float)(-2.0 * scale * st);
        }
    }
}

__global__ void f64_to_f32_kernel(const double* __restrict__ a, float* b, uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

int adj_check(const fbp_dims* d, const float* V, const float* T, const uint32_t* idx, const uint32_t* lab,
              const float* amp, const float* tau, uint32_t n)
{
    if (!d) return fail(FBP_E_ARG, "null dims");
    if (d->n_chans == 0 || d->n_samples == 0 || d->n_templates == 0 || d->template_len == 0)
        return fail(FBP_E_ARG, "invalid dims");
    if ((size_t)d->n_chans * (d->template_len + 2) * sizeof(double) > 200 * 1024)
        return fail(FBP_E_ARG, "channels x template length too large for one residual tile");
    if (!V || !T) return fail(FBP_E_ARG, "null pointer argument");
    if (n > 0 && (!idx || !lab || !amp || !tau)) return fail(FBP_E_ARG, "null spike argument");
    return FBP_OK;
}

AdjArgs adj_args(const fbp_dims* d, const float* V, const float* T, const uint32_t* idx, const uint32_t* lab,
                 const float* amp, const float* tau, uint32_t n)
{
    AdjArgs A;
    A.C = d->n_chans;
    A.N = d->n_samples;
    A.M = d->n_templates;
    A.W = d->template_len;
    A.V = V;
    A.T = T;
    A.idx = idx;
    A.lab = lab;
    A.amp = amp;
    A.tau = tau;
    A.n = n;
    return A;
}

}  // namespace
}  // namespace fbp

using namespace fbp;

extern "C" int fbp_adjoint_loss(const fbp_dims* dims, const float* voltage, const float* templates,
                                const uint32_t* spike_idx, const uint32_t* spike_lab, const float* amplitude,
                                const float* shift, uint32_t n_spikes, double* loss, void* stream)
{
    set_error("");
    const int rc = adj_check(dims, voltage, templates, spike_idx, spike_lab, amplitude, shift, n_spikes);
    if (rc != FBP_OK) return rc;
    if (!loss) return fail(FBP_E_ARG, "null loss");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const AdjArgs A = adj_args(dims, voltage, templates, spike_idx, spike_lab, amplitude, shift, n_spikes);
    FBP_CUDA(cudaMemsetAsync(loss, 0, sizeof(double), st));
    count_launch();
    const uint64_t nseg = ((uint64_t)A.N + kAdjSpan - 1) / kAdjSpan, most = 148ull * 16 * kAdjWarps;
    const uint32_t slices = (uint32_t)std::min<uint64_t>(A.C, std::max<uint64_t>(1, most / nseg));
    const uint32_t blocks = (uint32_t)((std::min<uint64_t>(nseg * slices, most) + kAdjWarps - 1) / kAdjWarps);
    if (slices > 1)
        adjoint_loss_kernel<true><<<blocks, kAdjThreads, 0, st>>>(A, slices, loss);
    else
        adjoint_loss_kernel<false><<<blocks, kAdjThreads, 0, st>>>(A, 1, loss);
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

extern "C" int fbp_adjoint_grad(const fbp_dims* dims, const float* voltage, const float* templates,
                                const uint32_t* spike_idx, const uint32_t* spike_lab, const float* amplitude,
                                const float* shift, uint32_t n_spikes, double scale, double* grad_templates64,
                                float* grad_templates, float* grad_amplitude, float* grad_shift, void* stream)
{
    set_error("");
    const int rc = adj_check(dims, voltage, templates, spike_idx, spike_lab, amplitude, shift, n_spikes);
    if (rc != FBP_OK) return rc;
    if (!grad_templates64 || !grad_templates || (n_spikes && (!grad_amplitude || !grad_shift)))
        return fail(FBP_E_ARG, "null gradient output");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const AdjArgs A = adj_args(dims, voltage, templates, spike_idx, spike_lab, amplitude, shift, n_spikes);
    const uint64_t nt = (uint64_t)A.M * A.C * A.W;
    FBP_CUDA(cudaMemsetAsync(grad_templates64, 0, nt * sizeof(double), st));
    if (n_spikes) {
        count_launch();
        const uint32_t blocks = std::min(n_spikes, 148u * 16);
        if (A.C > 8 && n_spikes <= 148u * 4)
            adjoint_grad_kernel<16><<<blocks, 32 * 16, 0, st>>>(A, scale, grad_templates64, grad_amplitude, grad_shift);
        else
            adjoint_grad_kernel<4><<<blocks, 32 * 4, 0, st>>>(A, scale, grad_templates64, grad_amplitude, grad_shift);
    }
    count_launch();
    f64_to_f32_kernel<<<148 * 4, 256, 0, st>>>(grad_templates64, grad_templates, nt);
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}
