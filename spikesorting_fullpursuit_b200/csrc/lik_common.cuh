// lik_common.cuh -- what the fast likelihood kernels (corr_fft.cu, lik_tc.cu) share:
// window maximum keys and the exact recomputation of single samples.
#pragma once

#include "fbp_internal.cuh"

namespace fbp {

// Key of a positive likelihood v at (template t, sample s) of window w:
// larger for a larger value, then for a smaller t, then for a smaller s -- the
// order in which compute_template_maximum_likelihood (binary_pursuit.cl:395-408)
// keeps the first maximum.  Needs W <= 1024 and t < 2^22.
__device__ __forceinline__ unsigned long long window_key(float v, uint32_t t, uint32_t local_s)
{
    return ((unsigned long long)__float_as_uint(v) << 32) | (unsigned long long)(0xFFFFFFFFu - ((t << 10) | local_s));
}

// The reference's sum, skipping template channels that are entirely zero
// (tnorm == 0): there it adds 0 * v terms, which leave a nonzero sum unchanged
// (and a zero sum zero, up to the sign of zero, which no decision reads).
static __device__ float exact_likelihood(const Dims& d, const float* __restrict__ V, const float* __restrict__ T,
                                         float b, uint32_t t, uint32_t s, const float* __restrict__ tnorm)
{
    float acc = b;
    for (uint32_t c = 0; c < d.C; ++c) {
        if (tnorm[(uint64_t)t * d.C + c] == 0.f) continue;
        const float* tr = T + ((uint64_t)t * d.C + c) * d.W;
        const float* vr = V + (uint64_t)c * d.N + s;
        for (uint32_t j = 0; j < d.W; ++j) acc = __fadd_rn(acc, __fmul_rn(tr[j], vr[j]));
    }
    return acc;
}

// Exact likelihood of (t, s) in the reference order (compute_maximum_likelihood,
// binary_pursuit.cl:216-252) from the current voltage, by a whole warp: the lanes form
// the products of four blocks of 32 taps (each product rounds the same wherever it is
// formed) in shared memory, the operands of the next four on their way meanwhile, and
// every lane adds them in tap order.  Channels where the template is entirely zero add
// 0 * v terms in the reference, which leave a nonzero sum unchanged.
//
// With one block of 32 on its way, a value of 8 channels took the latency of 25 to 32
// loads one after the other; the overlap recheck's parse, two such values a window,
// took 24 us a pass (8 channels, 17 templates, 8 s) and takes 11.
constexpr int kExactBlocks = 4;

static __device__ float warp_exact_lik(const Dims& d, const float* __restrict__ V, const float* __restrict__ T, float b,
                                       uint32_t t, uint32_t s, const float* __restrict__ tnorm, float* buf)
{
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31, C = d.C, W = d.W;
    const float* tn = tnorm + (uint64_t)t * C;
    const float *tr = nullptr, *vr = nullptr;   // the channel's rows, at this lane
    uint32_t cb = 0, j0 = W;                    // first channel of `live`, first tap of the block
    uint32_t live = __ballot_sync(full, lane < C && tn[lane] != 0.f);
    float tv[kExactBlocks], vv[kExactBlocks];
    uint32_t n[kExactBlocks];
    bool more = true;
    auto fetch = [&]() {
#pragma unroll
        for (int q = 0; q < kExactBlocks; ++q) {
            n[q] = 0;
            if (!more) continue;
            j0 += 32;
            if (j0 >= W) {   // the next non-zero channel
                while (live == 0u && (cb += 32) < C) live = __ballot_sync(full, cb + lane < C && tn[cb + lane] != 0.f);
                if (live == 0u) {
                    more = false;
                    continue;
                }
                const uint32_t c = cb + __ffs(live) - 1;
                live &= live - 1;
                tr = T + ((uint64_t)t * C + c) * W + lane;
                vr = V + (uint64_t)c * d.N + s + lane;
                j0 = 0;
            }
            n[q] = min(W - j0, 32u);
            if (lane < n[q]) {
                tv[q] = __ldg(tr + j0);
                vv[q] = vr[j0];
            }
        }
    };
    float acc = b;
    fetch();
    while (n[0] != 0u) {
        uint32_t total = 0;
#pragma unroll
        for (int q = 0; q < kExactBlocks; ++q) {
            if (lane < n[q]) buf[total + lane] = __fmul_rn(tv[q], vv[q]);
            total += n[q];
        }
        __syncwarp();
        fetch();
        uint32_t i = 0;
        for (; i + 16 <= total; i += 16) {
#pragma unroll
            for (int k = 0; k < 16; ++k) acc = __fadd_rn(acc, buf[i + k]);
        }
        for (; i < total; ++i) acc = __fadd_rn(acc, buf[i]);
        __syncwarp();
    }
    return acc;
}

// With lazy exactness, each positive exact value also enters its window's key
// and positive flag (after the likelihood kernel has published the CTA's own).
__device__ __forceinline__ void note_window(const Dims& d, unsigned long long* wkey, uint8_t* wpos, float v,
                                            uint32_t t, uint32_t s)
{
    if (wkey == nullptr || !(v > 0.f)) return;
    const uint32_t w = s / d.W;
    atomicMax(&wkey[w], window_key(v, t, s - w * d.W));
    wpos[w] = 1;
}

}  // namespace fbp
