// Index arithmetic of the tensor-core filter (filter.cu) that its host plan and
// its kernels share.  No CUDA types: a host compiler can walk the plan too.
#pragma once

#include <stdint.h>

#ifndef PQ_PLAN
#ifdef __CUDACC__
#define PQ_PLAN __host__ __device__ __forceinline__
#else
#define PQ_PLAN inline
#endif
#endif

namespace pq {

constexpr uint32_t FILTER_TILE = 128;         // candidates per tile
constexpr uint32_t FILTER_MAX_CHUNKS = 2048;  // chunk maxima per query the bound kernel holds

// Pass 1 keeps the maximum of every chunk of 2^logc columns of a query's row.
// Up to 64 columns a tile holds whole chunks, numbered in column order.  From
// 128 columns on a chunk is the tiles of one parity (they belong to one group
// of epilogue warps) among 2^(logc - 6) neighbours: the maximum is stored at
// the last of them in the job, at this place.
PQ_PLAN uint32_t filter_chunk_slot(uint32_t tile, uint32_t logc) {
    return ((tile >> 1) >> (logc - 7)) * 2 + (tile & 1u);
}
PQ_PLAN bool filter_chunk_ends(uint32_t tile, uint32_t job_end, uint32_t logc) {
    return (((tile >> 1) + 1) & ((1u << (logc - 7)) - 1u)) == 0 || tile + 2 >= job_end;
}

// Chunk maxima per query: every one of them is written.  (The wide chunks come
// in pairs, an even and an odd one; a last pair of a single tile has no odd one,
// whose place, the last, would keep whatever the workspace held.)
PQ_PLAN uint32_t filter_chunk_count(uint32_t tiles, uint32_t logc) {
    if (logc < 7) return tiles << (7 - logc);
    const uint32_t ct = 1u << (logc - 6);
    return 2 * ((tiles + ct - 1) / ct) - (tiles % ct == 1 ? 1 : 0);
}

// The widest power-of-two chunk (at least 8 columns) that still leaves 4 ksel
// chunks (the bound then admits about 15 % more than ksel points), and at most
// FILTER_MAX_CHUNKS of them.
PQ_PLAN uint32_t filter_chunk_log(uint32_t n, uint32_t tiles, uint32_t ksel) {
    const uint64_t want = 4 * ksel > 64 ? 4 * ksel : 64;
    uint32_t lc = 3;
    while ((uint64_t(n) >> (lc + 1)) >= want) ++lc;
    while (filter_chunk_count(tiles, lc) > FILTER_MAX_CHUNKS) ++lc;
    return lc;
}

// The admission margin, in units of s^2 = (|q| + sqrt(D))^2, and the error of an
// approximate squared distance in them that it has to cover twice (filter.cu).
constexpr float FILTER_MARGIN = 3.0f / 16384.0f;
constexpr double FILTER_ERROR_SPLIT = 1.0 / 16384.0;  // the BF16 parts, in |q| |x| <= s^2
constexpr double FILTER_ERROR_SUMS = 2.6e-5;          // the FP32 norms and the accumulator

// Tiles per job when a query block's candidates are cut into at most `want`
// slices: whole chunks, and at least two tiles.
PQ_PLAN uint32_t filter_slice_tiles(uint32_t tiles, uint32_t logc, uint32_t want) {
    const uint32_t ct = logc > 6 ? 1u << (logc - 6) : 1u;
    const uint32_t most = tiles / 2 < want ? tiles / 2 : want, sl = most > 1 ? most : 1;
    return ((tiles + sl - 1) / sl + ct - 1) / ct * ct;
}

}  // namespace pq
