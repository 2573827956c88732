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
// binary_pursuit.cl:216-252) from the current voltage, by a whole warp: each
// lane forms the products of 32 taps at a time (each product rounds the same
// wherever it is formed), the operands of the next 32 on their way meanwhile,
// and every lane adds them in tap order, so all lanes end with the reference's
// sum.  Channels where the template is entirely zero add 0 * v terms in the
// reference, which leave a nonzero sum unchanged.
static __device__ float warp_exact_lik(const Dims& d, const float* __restrict__ V, const float* __restrict__ T, float b,
                                       uint32_t t, uint32_t s, const float* __restrict__ tnorm)
{
    const uint32_t full = 0xffffffffu, lane = threadIdx.x & 31, C = d.C, W = d.W;
    float acc = b;
    const float* tn = tnorm + (uint64_t)t * C;
    for (uint32_t cb = 0; cb < C; cb += 32) {
        uint32_t live = __ballot_sync(full, cb + lane < C && tn[cb + lane] != 0.f);
        const float* tr = nullptr;
        const float* vr = nullptr;
        auto channel = [&]() {   // the next live channel's rows
            const uint32_t c = cb + __ffs(live) - 1;
            live &= live - 1;
            tr = T + ((uint64_t)t * C + c) * W;
            vr = V + (uint64_t)c * d.N + s;
        };
        bool more = live != 0u;
        uint32_t j0 = 0;
        float tv = 0.f, vv = 0.f;
        if (more) {
            channel();
            if (lane < W) {
                tv = __ldg(tr + lane);
                vv = vr[lane];
            }
        }
        while (more) {
            const float p = __fmul_rn(tv, vv);
            const uint32_t n = W - j0 < 32u ? W - j0 : 32u;
            j0 += 32;
            if (j0 >= W) {
                more = live != 0u;
                j0 = 0;
                if (more) channel();
            }
            tv = 0.f;
            vv = 0.f;
            if (more && j0 + lane < W) {
                tv = __ldg(tr + j0 + lane);
                vv = vr[j0 + lane];
            }
            if (n == 32u) {
#pragma unroll
                for (uint32_t k = 0; k < 32; ++k) acc = __fadd_rn(acc, __shfl_sync(full, p, k));
            } else {
#pragma unroll 8
                for (uint32_t k = 0; k < n; ++k) acc = __fadd_rn(acc, __shfl_sync(full, p, k));
            }
        }
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
