// pair_rule.cuh -- which kernel pairwise separability takes (separability.cu).
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifndef __CUDACC__   // a plain C++ program can ask the rule too
#define __host__
#define __device__
#endif

namespace fbp {

constexpr uint32_t kTilePairs = 64;   // pairs of a tile

struct PairTileSmem {
    size_t k, d, t1, nz, total;   // byte offsets; total
};

// zeros before and after template n1: the lags, in whole groups of 16, and a channel's
// last 32 lanes reach past it (by at most max_shift + 15 + 31, max_shift < W)
__host__ __device__ inline uint32_t pair_pad(uint32_t W) { return W + 48; }

// shared memory of a tile whose lanes take nj columns each
__host__ __device__ inline PairTileSmem pair_tile_smem(uint32_t nj, uint32_t C, uint32_t W)
{
    PairTileSmem s;
    s.k = 0;                                                     // [2][W][8 nj] covariances, zero columns past W
    s.d = s.k + (size_t)2 * W * 8 * nj * 8;                      // [64][8 nj] aligned differences
    s.t1 = s.d + (size_t)kTilePairs * 8 * nj * 8;                // [C W] template n1 between zeros
    s.nz = s.t1 + ((size_t)C * W + 2 * pair_pad(W)) * 8;          // [65][C] non-zero channels of the n2, then of n1
    s.total = s.nz + (size_t)(kTilePairs + 1) * C;
    return s;
}

// Whether tiles are faster than a CTA per pair.  A tile's CTA goes through the channels one
// after the other, so few units leave most SMs idle, and short windows give it little to do
// between two barriers.  Measured (us, CTA per pair / tiles; units zero on all but six
// channels, and without a zero channel from 24 units on where the two differ):
//   64 channels x 76 samples: 12 units 87 / 446, 48 479 / 628, 60 712 / 691, 80 1206 / 858
//                             (dense 24 1099 / 913, 60 5078 / 1852)
//   32 x 76: 40 251 / 347, 60 509 / 425;   16 x 76: 40 214 / 235, 44 273 / 249
//   10 x 76: 40 194 / 188;   4 x 76: 60 137 / 144, 72 184 / 152;   4 x 101: 60 222 / 223
//   16 x 61: 52 177 / 198, 60 229 / 211;   4 x 61: 64 95 / 101, 72 115 / 101
//   16 x 46: 80 231 / 241, 128 540 / 359;   64 x 32: 112 516 / 569, 128 666 / 566
//   16 x 24: 112 169 / 188, 200 493 / 460;   64 x 16: 200 units 390 / 700;   16 x 8: 140 / 299
// Dense sets of 24 to 63 units on more than 24 channels would gain from tiles too, but
// their zero channels are not known here.
__host__ __device__ inline bool pair_tiles_pay(uint32_t M, uint32_t C, uint32_t W)
{
    if (W < 56) return W >= 32 && M >= 2 * kTilePairs;
    return M >= (C >= 8 && C <= 24 && W >= 70 ? 48u : kTilePairs);
}

// Columns a lane of the tile kernel takes (8 lanes hold a row: W <= 8 of them), or 0: a CTA
// per pair, also where a template and two covariances do not fit `most` bytes of shared
// memory.  In 227 KB they fit up to 225 channels at W = 64, 133 at 76, 120 at 80, 18 at 96,
// 7 at 101 and 1 at 104, and from 105 on (14 columns or more) never.
__host__ __device__ inline uint32_t pair_tile_columns(uint32_t M, uint32_t C, uint32_t W, size_t most)
{
    if (!pair_tiles_pay(M, C, W)) return 0;
    const uint32_t cols[] = {8, 10, 13};
    for (uint32_t nj : cols)
        if (W <= 8 * nj && pair_tile_smem(nj, C, W).total + 2048 <= most) return nj;
    return 0;
}

}  // namespace fbp
