// compact.cuh -- ordered stream compaction in one launch.
//
// A functor supplies visit(i), which evaluates item i once and says whether it is kept,
// and emit(i, pos).  Tiles are numbered by a ticket, so that every tile before one that
// runs has started; a tile publishes its count, then adds up the counts of the tiles
// before it, back to the nearest one that knows its own position (decoupled look-back).
// (Count, scan and scatter as three launches took three times the launch gaps, and
// evaluated every item twice.)
//
// The wait for a predecessor is limited.  Past it the tile sets the error word, emits
// nothing and publishes that it failed; a tile that finds a failed one before it fails
// too, and a failed last tile leaves a total of 0.
#pragma once

#include <cub/cub.cuh>

#include "fbp_internal.cuh"

namespace fbp {

constexpr int kCompactThreads = 256;
constexpr int kCompactItems = 4;
constexpr int kCompactTile = kCompactThreads * kCompactItems;
constexpr uint32_t kLookbackPolls = 1u << 22;

// states of a tile: 0 (nothing yet), its count, its position past the tile, failed
constexpr unsigned long long kTileCount = 1ull << 62, kTilePlace = 2ull << 62, kTileFailed = 3ull << 62,
                             kTileFlags = 3ull << 62;

template <class F>
__global__ void __launch_bounds__(kCompactThreads) compact_kernel(F f, uint32_t n, unsigned long long* state,
                                                                  uint32_t* ticket, uint32_t* total, DevStatus* status,
                                                                  uint32_t polls_most)
{
    typedef cub::BlockScan<uint32_t, kCompactThreads> S;
    __shared__ typename S::TempStorage tmp;
    __shared__ uint32_t s_tile, s_base;
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const uint64_t first = (uint64_t)tile * kCompactTile + threadIdx.x * kCompactItems;
    bool keep[kCompactItems];
    uint32_t cnt = 0;
#pragma unroll
    for (int r = 0; r < kCompactItems; ++r) {
        keep[r] = first + r < n && f.visit((uint32_t)(first + r));
        cnt += keep[r];
    }
    uint32_t ex, all;
    S(tmp).ExclusiveSum(cnt, ex, all);
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        volatile unsigned long long* st = state;
        if (lane == 0) st[tile] = (tile ? kTileCount : kTilePlace) | all;
        uint32_t base = 0;
        bool failed = false;
        for (int64_t at = (int64_t)tile - 1; at >= 0;) {   // 32 predecessors at a time, nearest on lane 0
            const int64_t mine = at - lane;
            unsigned long long v = kTilePlace;
            if (mine >= 0) {
                uint32_t polls = 0;
                while (((v = st[mine]) & kTileFlags) == 0ull && ++polls < polls_most) {}
            }
            const unsigned long long flags = v & kTileFlags;
            const uint32_t place = __ballot_sync(0xffffffffu, flags == kTilePlace);
            const uint32_t upto = place ? (uint32_t)__ffs(place) - 1u : 31u;   // counts before it, and its position
            failed = __any_sync(0xffffffffu, lane <= upto && (flags == 0ull || flags == kTileFailed));
            if (failed) break;
            base += __reduce_add_sync(0xffffffffu, lane <= upto ? (uint32_t)v : 0u);
            if (place) break;
            at -= 32;
        }
        if (lane == 0) {
            if (failed) atomicOr(&status->error, 0x400u);
            st[tile] = failed ? kTileFailed : kTilePlace | (base + all);
            s_base = failed ? 0xFFFFFFFFu : base;
            if ((uint64_t)(tile + 1) * kCompactTile >= n) *total = failed ? 0u : base + all;
        }
    }
    __syncthreads();
    if (s_base == 0xFFFFFFFFu) return;
    uint32_t pos = s_base + ex;
#pragma unroll
    for (int r = 0; r < kCompactItems; ++r)
        if (keep[r]) f.emit((uint32_t)(first + r), pos++);
}

}  // namespace fbp
