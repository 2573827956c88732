// pairwise.cuh -- the order of numpy's pairwise summation: a range of more than 128
// values is split in two at a multiple of 8, depth first; a piece of at most 128 is
// summed with 8 partial sums (fewer than 8 values in order).
#pragma once

#include <stdint.h>

namespace fbp {

constexpr uint32_t kPairwisePiece = 128;

__host__ __device__ __forceinline__ uint32_t pairwise_split(uint32_t n)
{
    const uint32_t n2 = n / 2;
    return n2 - n2 % 8;
}

// Sum over [0, n) from the sums of its pieces, piece(first, count), taken left to right.
// A loop with its own stack (a range of 2^31 values is split 24 times deep): recursion
// would outgrow the 1 KB a device thread's calls get by default.
#pragma nv_exec_check_disable
template <class F, class Piece, class Add>
__host__ __device__ F pairwise_sum(uint32_t n, Piece&& piece, Add&& add)
{
    uint32_t first[26], count[26];
    F left[26];
    uint8_t side[26];   // 0: new, 1: in its left half, 2: in its right half
    int top = 0;
    first[0] = 0;
    count[0] = n;
    side[0] = 0;
    F done{};
    while (top >= 0) {
        if (count[top] <= kPairwisePiece) {
            done = piece(first[top], count[top]);
            --top;
            continue;
        }
        const uint32_t n2 = pairwise_split(count[top]);
        if (side[top] == 2) {
            done = add(left[top], done);
            --top;
            continue;
        }
        const bool right = side[top] == 1;
        if (right) left[top] = done;
        side[top] = right ? 2 : 1;
        first[top + 1] = right ? first[top] + n2 : first[top];
        count[top + 1] = right ? count[top] - n2 : n2;
        ++top;
        side[top] = 0;
    }
    return done;
}

// The pieces of ranges of one length and the additions of their sums, in order: step k
// adds the sum at right[k] to the one at left[k] (made on the host, passed by value).
constexpr uint32_t kPieces = 256;   // pieces of 64 values at least: ranges of 16,384 fit
struct PieceList {
    uint16_t count;
    uint16_t first[kPieces + 1];
    uint8_t left[kPieces], right[kPieces];
};

inline PieceList make_pieces(uint32_t len)
{
    PieceList l{};
    uint32_t adds = 0;
    pairwise_sum<uint32_t>(   // a sum is the place of its leftmost piece
        len,
        [&](uint32_t at, uint32_t) {
            l.first[l.count] = (uint16_t)at;
            return (uint32_t)l.count++;
        },
        [&](uint32_t a, uint32_t b) {
            l.left[adds] = (uint8_t)a;
            l.right[adds++] = (uint8_t)b;
            return a;
        });
    l.first[l.count] = (uint16_t)len;
    return l;
}

#ifdef __CUDACC__
__device__ __forceinline__ float sum_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sum_rn(double a, double b) { return __dadd_rn(a, b); }

// Sum of value(i) over [0, n <= 128) in numpy's order by 8 lanes (lane j of the group `mask`:
// the values j, j + 8, ... of the whole eights, combined as a tree, then the rest in
// order); n < 8: in order.  The sum on every lane of the group.
template <class F, class Value>
__device__ __forceinline__ F piece_sum(Value&& value, uint32_t n, uint32_t j, uint32_t mask)
{
    const uint32_t n8 = n - n % 8;
    F r = 0;
    if (n8) {
        r = value(j);
#pragma unroll 8
        for (uint32_t i = 8 + j; i < n8; i += 8) r = sum_rn(r, value(i));
        r = sum_rn(r, __shfl_xor_sync(mask, r, 1));
        r = sum_rn(r, __shfl_xor_sync(mask, r, 2));
        r = sum_rn(r, __shfl_xor_sync(mask, r, 4));
    }
    for (uint32_t i = n8; i < n; ++i) r = sum_rn(r, value(i));
    return r;
}

#endif  // __CUDACC__

}  // namespace fbp
