// preprocess.cu -- the pursuit's inputs built on the device (full_binary_pursuit's pre-processing).
//
// full_binary_pursuit (spikesorting_fullpursuit/overlap/full_binary_pursuit.py:325-349)
// builds the pursuit's templates and noise model from the sorted spikes: per unit,
// its clips on all channels (get_clips, processing/clip_utils.py:501-632), a robust
// template (calculate_robust_template, clip_utils.py:202-248), and from all units'
// clip-minus-template residuals one noise covariance per channel
// (get_channel_covariance_matrix, full_binary_pursuit.py:863-923).  Here:
//   * gather_clips_kernel: clips[k][n*Wc + j] = V[chans[n]][ev[k] + w0 + j].
//   * robust_template_kernel: per clip sample (column) of n clips, in float32 as
//     numpy computes it: med = median(x); mad = median(|x - med|) / 0.6745;
//     the template is median(x[med - mad < x < med + mad]), or med if that set is
//     empty.  Medians are exact order statistics (the mean of the two middle
//     values for an even count, as np.median) of order-preserving integer keys.
//     Up to 2048 clips a warp keeps a column's keys in registers and finds the
//     middle one bit by bit; above, robust_template_large_kernel selects by radix
//     (4 passes of 8 bits over shared-memory histograms, 32 columns a CTA).
//   * covariance_kernel: per channel, the FP64 covariance (ddof 0) of the
//     selected residual rows' samples on that channel: column means, then centred
//     products.  numpy multiplies with BLAS, so covariances agree to FP64 rounding.
#include <cooperative_groups.h>

#include <algorithm>

#include "fbp_internal.cuh"

namespace fbp {
namespace {

__global__ void gather_clips_kernel(const float* __restrict__ V, uint64_t N, const uint32_t* __restrict__ chans,
                                    uint32_t nch, const int64_t* __restrict__ ev, uint32_t n, int32_t w0, uint32_t wc,
                                    float* clips)
{
    const uint64_t len = (uint64_t)nch * wc;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < (uint64_t)n * len;
         e += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = e / len, r = e - k * len;
        const uint32_t ci = (uint32_t)(r / wc), j = (uint32_t)(r - (uint64_t)ci * wc);
        const int64_t s = ev[k] + w0 + (int64_t)j;
        clips[e] = V[(uint64_t)chans[ci] * N + (uint64_t)s];
    }
}

// order-preserving key of a float (finite or infinite)
__device__ __forceinline__ uint32_t fkey(float x)
{
    const uint32_t u = __float_as_uint(x);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unkey(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

constexpr int kRtCols = 32;      // columns per CTA (one per lane)
constexpr int kRtThreads = 256;  // 8 warps over the rows

// What a selection ranks, per column: 0 = x, 1 = |x - med|, 2 = x restricted to
// (lo, hi) (strict bounds).
struct RtColumn {
    float med, lo, hi;
};

// k-th smallest key (0-based) of each lane's column among its candidates.
// All threads of the CTA call it; returns the key for the calling lane's column.
__device__ uint32_t select_kth(const float* __restrict__ clips, uint32_t n, uint32_t len, uint32_t col0, int mode,
                               const RtColumn* cols, const uint32_t* kth, uint32_t* hist, uint32_t* s_prefix,
                               uint32_t* s_k)
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (threadIdx.x < kRtCols) {
        s_prefix[threadIdx.x] = 0;
        s_k[threadIdx.x] = kth[threadIdx.x];
    }
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (uint32_t e = threadIdx.x; e < kRtCols * 256; e += blockDim.x) hist[e] = 0;
        __syncthreads();
        const uint32_t col = col0 + lane;
        const uint32_t prefix = s_prefix[lane];
        const uint32_t pmask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
        if (col < len) {
            const RtColumn c = cols[lane];
            for (uint32_t i = warp; i < n; i += nwarps) {
                const float x = clips[(uint64_t)i * len + col];
                float v = x;
                if (mode == 1) v = fabsf(__fsub_rn(x, c.med));
                if (mode == 2 && !(x > c.lo && x < c.hi)) continue;
                const uint32_t key = fkey(v);
                if ((key & pmask) != (prefix & pmask)) continue;
                atomicAdd(&hist[lane * 256 + ((key >> shift) & 0xFFu)], 1u);
            }
        }
        __syncthreads();
        if (threadIdx.x < kRtCols) {
            const uint32_t* h = hist + threadIdx.x * 256;
            uint32_t k = s_k[threadIdx.x], b = 0;
            for (; b < 255; ++b) {
                if (k < h[b]) break;
                k -= h[b];
            }
            s_k[threadIdx.x] = k;
            s_prefix[threadIdx.x] |= b << shift;
        }
        __syncthreads();
    }
    return s_prefix[lane];
}

// median of a column's candidates: the middle key, or the float32 mean of the two
// middle values (np.median -> np.mean of two float32 values)
__device__ float column_median(const float* __restrict__ clips, uint32_t n, uint32_t len, uint32_t col0, int mode,
                               RtColumn* cols, uint32_t* cnt, uint32_t* kth, uint32_t* hist, uint32_t* s_prefix,
                               uint32_t* s_k)
{
    const uint32_t lane = threadIdx.x & 31;
    if (threadIdx.x < kRtCols) kth[threadIdx.x] = cnt[threadIdx.x] > 0 ? (cnt[threadIdx.x] - 1) / 2 : 0;
    __syncthreads();
    const float a = unkey(select_kth(clips, n, len, col0, mode, cols, kth, hist, s_prefix, s_k));
    __syncthreads();
    if (threadIdx.x < kRtCols) kth[threadIdx.x] = cnt[threadIdx.x] / 2;
    __syncthreads();
    const float b = unkey(select_kth(clips, n, len, col0, mode, cols, kth, hist, s_prefix, s_k));
    __syncthreads();
    const uint32_t c = cnt[lane];
    return (c & 1u) ? a : __fdiv_rn(__fadd_rn(a, b), 2.0f);
}

__global__ void __launch_bounds__(kRtThreads) robust_template_large_kernel(const float* __restrict__ clips,
                                                                           uint32_t n, uint32_t len, float* tmpl)
{
    __shared__ uint32_t hist[kRtCols * 256];
    __shared__ uint32_t s_prefix[kRtCols], s_k[kRtCols], kth[kRtCols], cnt[kRtCols];
    __shared__ RtColumn cols[kRtCols];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t col0 = blockIdx.x * kRtCols, col = col0 + lane;
    if (threadIdx.x < kRtCols) {
        cnt[threadIdx.x] = n;
        cols[threadIdx.x] = RtColumn{0.f, 0.f, 0.f};
    }
    __syncthreads();
    const float med = column_median(clips, n, len, col0, 0, cols, cnt, kth, hist, s_prefix, s_k);
    if (threadIdx.x < kRtCols) cols[threadIdx.x].med = med;
    __syncthreads();
    const float mad = __fdiv_rn(column_median(clips, n, len, col0, 1, cols, cnt, kth, hist, s_prefix, s_k), 0.6745f);
    if (threadIdx.x < kRtCols) {
        cols[threadIdx.x].lo = __fsub_rn(med, mad);
        cols[threadIdx.x].hi = __fadd_rn(med, mad);
        cnt[threadIdx.x] = 0;
    }
    __syncthreads();
    // size of the within-1-MAD set per column
    if (col < len) {
        const RtColumn c = cols[lane];
        uint32_t m = 0;
        for (uint32_t i = warp; i < n; i += blockDim.x >> 5) {
            const float x = clips[(uint64_t)i * len + col];
            m += (x > c.lo && x < c.hi) ? 1u : 0u;
        }
        atomicAdd(&cnt[lane], m);
    }
    __syncthreads();
    const float sel = column_median(clips, n, len, col0, 2, cols, cnt, kth, hist, s_prefix, s_k);
    if (threadIdx.x < kRtCols && col < len) tmpl[col] = cnt[threadIdx.x] > 0 ? sel : med;
}

// Median of the `cnt` valid keys of a warp's column (lane slots, 0xFFFFFFFF where
// there is none): the middle key bit by bit -- the largest value with at most k
// smaller keys -- and, for an even count, the next one.  Once at most 32 keys agree
// with the bits found, they go to the lanes and a step is one ballot instead of NV
// compares a lane: for 512 to 1024 clips 51 -> 29 us a unit of 1616 samples, for 1024
// to 2048, held back by its registers, 89 -> 85 us.  `few`: the warp's 32 words.
template <int NV>
__device__ __forceinline__ float warp_median(const uint32_t (&key)[NV], uint32_t cnt, uint32_t* few)
{
    const uint32_t full = 0xffffffffu, k = cnt > 0 ? (cnt - 1) / 2 : 0u, lane = threadIdx.x & 31;
    uint32_t a = 0, base = 0, top = cnt;   // [base, top): ranks of the keys that agree with a so far
    int bit = 31;
    for (; bit >= 0 && top - base > 32; --bit) {
        const uint32_t cand = a | (1u << bit);
        uint32_t below = 0;
#pragma unroll
        for (int i = 0; i < NV; ++i) below += key[i] < cand ? 1u : 0u;
        below = __reduce_add_sync(full, below);
        if (below <= k) {
            a = cand;
            base = below;
        } else {
            top = below;
        }
    }
    if (bit >= 0) {   // at most 32 left: one a lane for the remaining bits
        uint32_t n = 0;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const bool in = key[i] >= a && (key[i] - a) >> bit <= 1u && key[i] != 0xFFFFFFFFu;
            const uint32_t m = __ballot_sync(full, in);
            if (in) few[n + __popc(m & ((1u << lane) - 1u))] = key[i];
            n += __popc(m);
        }
        __syncwarp();
        const uint32_t mine = lane < n ? few[lane] : 0xFFFFFFFFu;
        __syncwarp();
        for (; bit >= 0; --bit) {
            const uint32_t cand = a | (1u << bit);
            if (base + __popc(__ballot_sync(full, mine < cand)) <= k) a = cand;
        }
    }
    if (cnt & 1u) return unkey(a);
    uint32_t upto = 0, next = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        upto += key[i] <= a ? 1u : 0u;
        next = key[i] > a && key[i] < next ? key[i] : next;
    }
    upto = __reduce_add_sync(full, upto);
    next = __reduce_min_sync(full, next);
    return __fdiv_rn(__fadd_rn(unkey(a), unkey(upto > cnt / 2 ? a : next)), 2.0f);
}

// A warp per column, n <= 32 NV clips in registers (8 adjacent columns a CTA: the
// 32-byte sectors of the clips are read once).  Three selections over NV keys a lane
// bound it.  40 units of about 600 clips x 1616 samples: 27.7 ms by radix selection
// from memory, 1616 / 32 CTAs a unit, against 1.4 ms.
template <int NV>
__global__ void __launch_bounds__(kRtThreads) robust_template_kernel(const float* __restrict__ clips, uint32_t n,
                                                                     uint32_t len, float* tmpl)
{
    __shared__ uint32_t few[kRtThreads / 32][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.x * (kRtThreads / 32) + warp;
    if (col >= len) return;
    float x[NV];
    uint32_t key[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const uint32_t r = i * 32 + lane;
        x[i] = r < n ? __ldg(clips + (uint64_t)r * len + col) : 0.f;
        key[i] = r < n ? fkey(x[i]) : 0xFFFFFFFFu;
    }
    const float med = warp_median<NV>(key, n, few[warp]);
#pragma unroll
    for (int i = 0; i < NV; ++i) key[i] = i * 32 + lane < n ? fkey(fabsf(__fsub_rn(x[i], med))) : 0xFFFFFFFFu;
    const float mad = __fdiv_rn(warp_median<NV>(key, n, few[warp]), 0.6745f);
    const float lo = __fsub_rn(med, mad), hi = __fadd_rn(med, mad);
    uint32_t cnt = 0;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const bool in = i * 32 + lane < n && x[i] > lo && x[i] < hi;
        key[i] = in ? fkey(x[i]) : 0xFFFFFFFFu;
        cnt += in ? 1u : 0u;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const float sel = warp_median<NV>(key, cnt, few[warp]);
    if (lane == 0) tmpl[col] = cnt > 0 ? sel : med;
}

// Covariance of one channel (blockIdx.z) between two tiles of kCovTile of its samples
// (blockIdx.y), over the channel's selected residual rows (rows[c][0..n_rows)):
// residual row r = clips[rows[r]] - template[unit[rows[r]]] in float32, then FP64.
// One pass: products and sums of x - s, s the mean of the first rows (at most
// kCovProbe), give sum (x - s)(y - s) - sum (x - s) sum (y - s) / n; s lies within a
// fraction of a standard deviation of the mean, so nothing cancels.  A cluster shares
// the rows; a thread accumulates 7 x 7 of the tile (on the diagonal only its upper
// 16-blocks) while the next rows are on their way, and the CTAs' parts are added in
// rank order through shared memory.  16 channels x 101 samples x 10,000 rows: 7.5 ms
// with the means summed by every output row's CTA, one scattered load at a time,
// 1.9 ms with a pass of its own for them, 0.5 ms now.
constexpr uint32_t kCovTile = 112, kCovRows = 16, kCovCluster = 8, kCovThreads = 256, kCovProbe = 32,
                   kCovFewRows = 64;
constexpr uint32_t kCovLoads = kCovRows * kCovTile / kCovThreads;   // elements of a step a thread loads

template <bool DIAG>
__global__ void __launch_bounds__(kCovThreads, 1)
    covariance_kernel(const float* __restrict__ clips, const float* __restrict__ tmpls,
                      const uint32_t* __restrict__ unit_of, const int64_t* __restrict__ rows, uint32_t n_rows,
                      uint32_t len, uint32_t wc, double* cov)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) double csm[];
    constexpr uint32_t kTiles = DIAG ? 1 : 2;
    double* part = csm;                              // [kCovTile][kCovTile] this CTA's products
    double* xs = part + kCovTile * kCovTile;         // [kTiles][kCovRows][kCovTile] rows of a step
    double* sums = xs + 2 * kCovRows * kCovTile;     // [2][kCovTile] this CTA's sums
    double* shift = sums + 2 * kCovTile;             // [2][kCovTile] s
    double* total = shift + 2 * kCovTile;            // [2][kCovTile] the cluster's sums
    __shared__ uint64_t s_clip[2][kCovRows], s_tmpl[2][kCovRows];   // row offsets of two steps
    const uint32_t nt = (wc + kCovTile - 1) / kCovTile, c = blockIdx.z, rank = cluster.block_rank(),
                   ctas = cluster.num_blocks();
    // tile pair: the diagonal launch numbers the tiles, the other one the ordered pairs
    const uint32_t it = DIAG ? blockIdx.y : blockIdx.y / (nt - 1);
    uint32_t jt = DIAG ? it : blockIdx.y % (nt - 1);
    if (!DIAG && jt >= it) ++jt;
    const uint32_t base[2] = {it * kCovTile, jt * kCovTile};
    const uint32_t cols[2] = {min(kCovTile, wc - base[0]), min(kCovTile, wc - base[1])};
    // whole steps a CTA; the last ones of a cluster have no rows if there are few
    const uint32_t share = max((n_rows + ctas - 1) / ctas, kCovRows), parts = (n_rows + share - 1) / share;
    const uint32_t r0 = min(n_rows, rank * share), r1 = min(n_rows, r0 + share);
    const int64_t* mine = rows + (uint64_t)c * n_rows;
    // provisional means
    const uint32_t probe = min(n_rows, kCovProbe);
    __shared__ uint64_t s_probe[2][kCovProbe];   // offsets of their clip and template
    if (threadIdx.x < probe) {
        const uint64_t row = (uint64_t)__ldg(mine + threadIdx.x);
        s_probe[0][threadIdx.x] = row * len + (uint64_t)c * wc;
        s_probe[1][threadIdx.x] = (uint64_t)__ldg(unit_of + row) * len + (uint64_t)c * wc;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kTiles * kCovTile; k += kCovThreads) {
        const uint32_t w = k / kCovTile, j = k - w * kCovTile;
        double s = 0.0;
        if (j < cols[w])
#pragma unroll 16
            for (uint32_t r = 0; r < probe; ++r)
                s += (double)__fsub_rn(__ldg(clips + s_probe[0][r] + base[w] + j), __ldg(tmpls + s_probe[1][r] + base[w] + j));
        shift[k] = s / (double)probe;
    }
    auto offsets = [&](uint32_t step) {   // row offsets of a step, by its first threads
        const uint32_t r = r0 + step * kCovRows + threadIdx.x;
        if (threadIdx.x < kCovRows && r < r1) {
            const uint64_t row = (uint64_t)__ldg(mine + r);
            s_clip[step & 1u][threadIdx.x] = row * len + (uint64_t)c * wc;
            s_tmpl[step & 1u][threadIdx.x] = (uint64_t)__ldg(unit_of + row) * len + (uint64_t)c * wc;
        }
    };
    float xv[kTiles][kCovLoads], tv[kTiles][kCovLoads];
    auto fetch = [&](uint32_t step) {     // a step's values into registers
#pragma unroll
        for (uint32_t w = 0; w < kTiles; ++w)
#pragma unroll
            for (uint32_t q = 0; q < kCovLoads; ++q) {
                const uint32_t e = threadIdx.x + q * kCovThreads, r = e / kCovTile, k = e - r * kCovTile;
                const bool in = r0 + step * kCovRows + r < r1 && k < cols[w];
                xv[w][q] = in ? __ldg(clips + s_clip[step & 1u][r] + base[w] + k) : 0.f;
                tv[w][q] = in ? __ldg(tmpls + s_tmpl[step & 1u][r] + base[w] + k) : 0.f;
            }
    };
    const uint32_t steps = (r1 - r0 + kCovRows - 1) / kCovRows;
    offsets(0);
    __syncthreads();   // the provisional means too
    if (steps > 0) fetch(0);
    const uint32_t tx = threadIdx.x & 15u, ty = threadIdx.x >> 4;
    double acc[7][7], sum = 0.0;
#pragma unroll
    for (int a = 0; a < 7; ++a)
#pragma unroll
        for (int b = 0; b < 7; ++b) acc[a][b] = 0.0;
    for (uint32_t st = 0; st < steps; ++st) {
        const uint32_t nr = min(kCovRows, r1 - (r0 + st * kCovRows));
#pragma unroll
        for (uint32_t w = 0; w < kTiles; ++w)
#pragma unroll
            for (uint32_t q = 0; q < kCovLoads; ++q) {
                const uint32_t e = threadIdx.x + q * kCovThreads, r = e / kCovTile, k = e - r * kCovTile;
                xs[w * kCovRows * kCovTile + e] =
                    r < nr && k < cols[w] ? (double)__fsub_rn(xv[w][q], tv[w][q]) - shift[w * kCovTile + k] : 0.0;
            }
        offsets(st + 1);
        __syncthreads();
        if (st + 1 < steps) fetch(st + 1);
        const double* second = DIAG ? xs : xs + kCovRows * kCovTile;
        for (uint32_t r = 0; r < nr; ++r) {
            double u[7], v[7];
#pragma unroll
            for (int a = 0; a < 7; ++a) {
                u[a] = xs[r * kCovTile + ty + 16 * a];
                v[a] = second[r * kCovTile + tx + 16 * a];
            }
#pragma unroll
            for (int a = 0; a < 7; ++a)
#pragma unroll
                for (int b = 0; b < 7; ++b)
                    if (!DIAG || b >= a) acc[a][b] = fma(u[a], v[b], acc[a][b]);
        }
        if (threadIdx.x < kTiles * kCovTile) {
            const uint32_t w = threadIdx.x / kCovTile, k = threadIdx.x - w * kCovTile;
            for (uint32_t r = 0; r < nr; ++r) sum += xs[(w * kCovRows + r) * kCovTile + k];
        }
        __syncthreads();
    }
    if (threadIdx.x < kTiles * kCovTile) sums[threadIdx.x] = sum;
    if (steps > 0) {
#pragma unroll
        for (int a = 0; a < 7; ++a)
#pragma unroll
            for (int b = 0; b < 7; ++b)
                if (!DIAG || b >= a) part[(ty + 16 * a) * kCovTile + tx + 16 * b] = acc[a][b];
    }
    cluster.sync();
    for (uint32_t k = threadIdx.x; k < kTiles * kCovTile; k += kCovThreads) {
        double s = 0.0;
        for (uint32_t b = 0; b < parts; ++b) s += cluster.map_shared_rank(sums, b)[k];
        total[k] = s;
    }
    __syncthreads();
    // this CTA's share of the tile, parts added in rank order
    const double inv = 1.0 / (double)n_rows;   // np.cov scales by 1 / fact
    for (uint32_t e = rank * kCovThreads + threadIdx.x; e < cols[0] * cols[1]; e += ctas * kCovThreads) {
        uint32_t i = e / cols[1], j = e - i * cols[1];
        const uint32_t oi = i, oj = j;
        if (DIAG && j < i) {   // the covariance is symmetric: only its upper 16-blocks are there
            i = oj;
            j = oi;
        }
        double s = 0.0;
        for (uint32_t b = 0; b < parts; ++b) s += cluster.map_shared_rank(part, b)[i * kCovTile + j];
        s -= (total[i] * total[(DIAG ? 0 : kCovTile) + j]) * inv;   // the same for (j, i)
        cov[((uint64_t)c * wc + base[0] + oi) * wc + base[1] + oj] = s * inv;
    }
    cluster.sync();   // no CTA leaves while another reads its part
}

}  // namespace
}  // namespace fbp

using namespace fbp;

extern "C" int fbp_gather_clips(const float* voltage, uint32_t n_chans, uint64_t n_samples, const uint32_t* chans,
                                uint32_t n_nbr, const int64_t* event_indices, uint32_t n, int32_t win0,
                                uint32_t win_len, float* clips, void* stream)
{
    set_error("");
    if (n == 0) return FBP_OK;
    if (!voltage || !chans || !event_indices || !clips || n_nbr == 0 || win_len == 0 || n_chans == 0)
        return fail(FBP_E_ARG, "invalid arguments");
    const uint64_t total = (uint64_t)n * n_nbr * win_len;
    const uint32_t grid = (uint32_t)std::min<uint64_t>((total + 255) / 256, 148ull * 32);
    gather_clips_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(voltage, n_samples, chans, n_nbr,
                                                                              event_indices, n, win0, win_len, clips);
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

extern "C" int fbp_robust_template(const float* clips, uint32_t n, uint32_t clip_len, float* tmpl, void* stream)
{
    set_error("");
    if (n == 0 || clip_len == 0) return fail(FBP_E_ARG, "no clips");
    if (!clips || !tmpl) return fail(FBP_E_ARG, "null pointer argument");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const uint32_t grid = (clip_len + kRtThreads / 32 - 1) / (kRtThreads / 32);
    if (n <= 256)
        robust_template_kernel<8><<<grid, kRtThreads, 0, st>>>(clips, n, clip_len, tmpl);
    else if (n <= 512)
        robust_template_kernel<16><<<grid, kRtThreads, 0, st>>>(clips, n, clip_len, tmpl);
    else if (n <= 1024)
        robust_template_kernel<32><<<grid, kRtThreads, 0, st>>>(clips, n, clip_len, tmpl);
    else if (n <= 2048)
        robust_template_kernel<64><<<grid, kRtThreads, 0, st>>>(clips, n, clip_len, tmpl);
    else   // more keys than a warp holds
        robust_template_large_kernel<<<(clip_len + kRtCols - 1) / kRtCols, kRtThreads, 0, st>>>(clips, n, clip_len, tmpl);
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}

extern "C" int fbp_residual_covariance(const float* clips, const float* templates, const uint32_t* unit_of,
                                       const int64_t* rows, uint32_t n_rows, uint32_t clip_len, uint32_t n_chans,
                                       uint32_t n_samples_per_chan, double* cov, void* stream)
{
    set_error("");
    if (n_rows == 0 || n_chans == 0 || n_samples_per_chan == 0) return fail(FBP_E_ARG, "invalid sizes");
    if ((uint64_t)n_chans * n_samples_per_chan > clip_len) return fail(FBP_E_ARG, "clip shorter than channels x samples");
    if (!clips || !templates || !unit_of || !rows || !cov) return fail(FBP_E_ARG, "null pointer argument");
    if ((size_t)n_samples_per_chan * 8 > 48 * 1024) return fail(FBP_E_ARG, "samples per channel too large");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t smem = (kCovTile * kCovTile + 2 * kCovRows * kCovTile + 6 * kCovTile) * sizeof(double);
    const uint32_t nt = (n_samples_per_chan + kCovTile - 1) / kCovTile;
    // few rows of many channels: a cluster a channel would be several waves of CTAs with a
    // step or none each (256 channels x 61 samples x 50 rows 186 us, by a CTA a channel 38)
    const uint32_t ctas = n_rows <= kCovFewRows && (uint64_t)n_chans * nt * kCovCluster > 148 ? 1 : kCovCluster;
    auto launch = [&](auto kernel, uint32_t tiles) -> cudaError_t {
        cudaError_t e = allow_max_dyn_smem(kernel);
        if (e != cudaSuccess) return e;
        cudaLaunchAttribute shape;
        shape.id = cudaLaunchAttributeClusterDimension;
        shape.val.clusterDim.x = ctas;
        shape.val.clusterDim.y = shape.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(ctas, tiles, n_chans);
        cfg.blockDim = dim3(kCovThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = &shape;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kernel, clips, templates, unit_of, rows, n_rows, clip_len, n_samples_per_chan, cov);
    };
    FBP_CUDA(launch(covariance_kernel<true>, nt));
    if (nt > 1) FBP_CUDA(launch(covariance_kernel<false>, nt * (nt - 1)));
    FBP_CUDA(cudaGetLastError());
    return FBP_OK;
}
