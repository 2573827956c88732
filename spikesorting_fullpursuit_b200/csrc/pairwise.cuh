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

}  // namespace fbp
