// fft256.cuh -- 256-point complex transforms by half-warps, and the template
// spectra they meet.
//
// A correlation of a short template with the voltage,
//     r[n] = sum_c sum_j T[c][j] v[c][n + j],
// is r = IDFT( sum_c conj(DFT(T[c])) DFT(v[c]) ).  Two real signals share one
// complex transform: with z = v_A + i v_B the product sum is r_A + i r_B, since
// the templates are real; nothing has to be separated in between.
//
// A half-warp holds one transform, 16 values a thread: thread l holds the inputs
// l, l + 16, ..., transforms them (16 = 4 x 4 in registers), multiplies by
// e^(+-2 pi i l r / 256), exchanges through 2 KB of shared memory (stored at
// column l ^ r of row r: rows are written and columns read without bank
// conflicts) and transforms again; it then holds outputs l, l + 16, ..., the same
// residue class it started from, which is the order the next step reads.
//
// Rounding, u = 2^-24, elementwise: each of the 8 additions a value goes through
// adds at most u, each of the 3 complex multiplications between them at most
// (sqrt 5 + 1) u (product, and the factor's own rounding), relative to the sum of
// the magnitudes of the inputs that reach the output: below 18 u per transform;
// 24 u is used.  The spectra are computed in FP64 and rounded once (u); a product
// sum over n channels adds at most 2 sqrt 2 n u.  By Cauchy-Schwarz and Parseval
// an output is off by at most
//     (2 * 24 + 1 + 2.83 n + 2) u  sum_c |T_c| |z_c|  <  (64 + 3 n) u sum_c |T_c| |z_c|
// (kFftTerms).  Channels where the template is all zero do not enter.
#pragma once

#include "fbp_internal.cuh"

namespace fbp {

constexpr uint32_t kFft = 256;          // transform length
constexpr float kFftTerms = 64.f;       // rounding of a correlation: (kFftTerms + 3 n) u, see above

// Template spectra, by the template's non-zero channels clist[t][0 .. ccnt[t]):
// spec[t][i][m][l] = {X(k), X(k + 16)}, k = l + 32 m, X = DFT(T[t][clist[t][i]]) / 256 (the
// inverse transform's scale), complex as {re, im}.
struct FftTables {
    const float4* spec;       // [M][C][8][16]
    const uint8_t* clist;     // [M][C]
    const uint32_t* ccnt;     // [M]
    const float2* tw;         // [16][16] e^(2 pi i l r / 256) at r * 16 + l
};

#ifdef __CUDACC__

__device__ __forceinline__ float2 c_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 c_sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// a * (wr + i wi)
__device__ __forceinline__ float2 c_mul(float2 a, float wr, float wi)
{
    return make_float2(fmaf(a.x, wr, -(a.y * wi)), fmaf(a.x, wi, a.y * wr));
}

// 4-point transform, exponent sign SG
template <int SG>
__device__ __forceinline__ void fft4(float2& a, float2& b, float2& c, float2& d)
{
    const float2 s0 = c_add(a, c), s1 = c_sub(a, c), s2 = c_add(b, d), e = c_sub(b, d);
    const float2 s3 = SG > 0 ? make_float2(-e.y, e.x) : make_float2(e.y, -e.x);   // SG i (b - d)
    a = c_add(s0, s2);
    b = c_add(s1, s3);
    c = c_sub(s0, s2);
    d = c_sub(s1, s3);
}

// 16-point transform in registers, outputs in order
template <int SG>
__device__ __forceinline__ void fft16(float2 (&x)[16])
{
    constexpr float c1 = 0.92387953251128674f, s1 = SG * 0.38268343236508977f, h = 0.70710678118654752f;
#pragma unroll
    for (int l = 0; l < 4; ++l) fft4<SG>(x[l], x[l + 4], x[l + 8], x[l + 12]);   // x[l + 4 r]
    x[5] = c_mul(x[5], c1, s1);
    x[9] = c_mul(x[9], h, SG * h);
    x[13] = c_mul(x[13], SG * s1, SG * c1);
    x[6] = c_mul(x[6], h, SG * h);
    x[10] = SG > 0 ? make_float2(-x[10].y, x[10].x) : make_float2(x[10].y, -x[10].x);
    x[14] = c_mul(x[14], -h, SG * h);
    x[7] = c_mul(x[7], SG * s1, SG * c1);
    x[11] = c_mul(x[11], -h, SG * h);
    x[15] = c_mul(x[15], -c1, -s1);
#pragma unroll
    for (int r = 0; r < 4; ++r) fft4<SG>(x[4 * r], x[4 * r + 1], x[4 * r + 2], x[4 * r + 3]);   // x[4 r + q] = output 4 q + r
    // to natural order: a 4 x 4 transposition of register names
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = r + 1; q < 4; ++q) {
            const float2 t = x[4 * r + q];
            x[4 * r + q] = x[4 * q + r];
            x[4 * q + r] = t;
        }
}

// 256-point transform of a half-warp (both half-warps of the warp call it
// together): x[m] = input l + 16 m -> x[q] = output l + 16 q.  buf: the
// half-warp's 256 float2 of shared memory; tw: FftTables::tw in shared memory.
template <int SG>
__device__ __forceinline__ void fft256(float2 (&x)[16], float2* buf, const float2* tw, uint32_t l)
{
    // one copy of the 16-point transform in the code, run twice: unrolled, the kernels
    // outgrow the instruction cache (a third of their stalls)
#pragma unroll 1
    for (int step = 0;; ++step) {
        fft16<SG>(x);
        if (step) return;
#pragma unroll
        for (uint32_t r = 0; r < 16; ++r) {
            if (r) {
                const float2 w = tw[r * 16 + l];
                x[r] = c_mul(x[r], w.x, SG * w.y);
            }
            buf[r * 16 + (l ^ r)] = x[r];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) x[i] = buf[l * 16 + (i ^ l)];
        __syncwarp();
    }
}

// Forward transform of channel data x (input order) into the channel's spectrum
// zs[8][16] (float4 {Z(k), Z(k + 16)}, k = l + 32 m): 2 KB, used for the exchange too.
__device__ __forceinline__ void fft_channel(float2 (&x)[16], float4* zs, const float2* tw, uint32_t l)
{
    fft256<-1>(x, reinterpret_cast<float2*>(zs), tw, l);
#pragma unroll
    for (uint32_t m = 0; m < 8; ++m) zs[m * 16 + l] = make_float4(x[2 * m].x, x[2 * m].y, x[2 * m + 1].x, x[2 * m + 1].y);
}

// One template of a half-warp, as far as it is fetched ahead of its use: its channel
// count, the channels of its first 16 list entries (entry l on lane l) and the first
// half of its first spectrum.
struct FftAhead {
    uint32_t cnt, cl;
    float4 T[4];
};

__device__ __forceinline__ void fft_fetch(const FftTables& F, uint32_t C, uint32_t t, bool valid, uint32_t l, FftAhead& A)
{
    A.cnt = valid ? __ldg(F.ccnt + t) : 0u;
    A.cl = valid && l < C ? F.clist[(size_t)t * C + l] : 0u;
    const float4* sp = F.spec + (size_t)t * C * 128 + l;
#pragma unroll
    for (int m = 0; m < 4; ++m) A.T[m] = valid ? __ldg(sp + m * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
}

__device__ __forceinline__ void fft_mac4(const float4 (&T)[4], const float4* zp, float2* x)
{
#pragma unroll
    for (int m = 0; m < 4; ++m) {   // x += conj(T) Z
        const float4 Z = zp[m * 16];
        x[2 * m].x = fmaf(T[m].x, Z.x, fmaf(T[m].y, Z.y, x[2 * m].x));
        x[2 * m].y = fmaf(T[m].x, Z.y, fmaf(-T[m].y, Z.x, x[2 * m].y));
        x[2 * m + 1].x = fmaf(T[m].z, Z.z, fmaf(T[m].w, Z.w, x[2 * m + 1].x));
        x[2 * m + 1].y = fmaf(T[m].z, Z.w, fmaf(-T[m].w, Z.z, x[2 * m + 1].y));
    }
}

// Correlation of template t (fetched ahead in A) with the channel spectra zs[C][8][16]
// of the CTA's signal pair, by a half-warp: x[q] = r_A[l + 16 q] + i r_B[l + 16 q].  A
// half-warp without a template has A.cnt == 0 (it takes part in the exchange).  The
// spectra come from L2: each half spectrum is loaded while the one before it is
// used, and template tn's first while t is transformed.
__device__ __forceinline__ void fft_correlate(const FftTables& F, uint32_t C, uint32_t t, FftAhead& A, uint32_t tn,
                                              bool next, const float4* zs, float2* buf, const float2* tw, uint32_t l,
                                              float2 (&x)[16])
{
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = make_float2(0.f, 0.f);
    const uint32_t cnt = A.cnt, half = 0xFFFFu << (threadIdx.x & 16u);
    const float4* sp = F.spec + (size_t)t * C * 128 + l;
    const float4* zl = zs + l;
    for (uint32_t i = 0; i < cnt; ++i) {
        if ((i & 15u) == 0u && i) A.cl = i + l < C ? F.clist[(size_t)t * C + i + l] : 0u;
        const float4* zp = zl + __shfl_sync(half, A.cl, i & 15u, 16) * 128;
        float4 B[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) B[m] = __ldg(sp + 64 + m * 16);
        fft_mac4(A.T, zp, x);
        sp += 128;
        if (i + 1 < cnt) {
#pragma unroll
            for (int m = 0; m < 4; ++m) A.T[m] = __ldg(sp + m * 16);
        }
        fft_mac4(B, zp + 64, x + 8);
    }
    __syncwarp();
    fft_fetch(F, C, next ? tn : 0u, next, l, A);
    fft256<1>(x, buf, tw, l);
}

// sum of v over the half-warp's 16 lanes, on every lane
__device__ __forceinline__ float half_sum(float v)
{
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

#endif  // __CUDACC__

}  // namespace fbp
