// Tensor-core filter of the exact searches (filter.cu): which points can be
// among a query's nearest, decided by bounds on split-BF16 distance
// tiles; the survivors get the search's own FP32 distances.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <functional>
#include <vector>

struct pq_ctx;

namespace pq {

// One group of points searched among themselves.
struct FilterSample {
    uint64_t base;    // first row
    uint64_t out;     // first output element
    uint64_t rcp;     // floor((2^64 - 1) / n)
    uint32_t n;       // points
    uint32_t k;       // nearest points wanted (EXACT: itself included)
    uint32_t ksel;    // chunk maxima the bound is taken from: k + 1
    uint32_t stride;  // candidate position p holds point p * stride mod n
    uint32_t inv;     // point j sits at position j * inv mod n
    uint32_t tiles;   // 128-candidate tiles
    uint32_t logc;    // log2 of the columns per chunk maximum
    uint32_t chunks;  // chunk maxima per query
    uint32_t slices;  // candidate ranges searched by separate jobs
    uint32_t cap;     // admitted candidates kept per (query, slice, tile parity)
};

enum { FILTER_BATCHED = 0, FILTER_EUCLIDEAN = 1, FILTER_COSINE = 2 };

// Points of a group the filter takes: enough that the chunk maxima bound the
// k-th distance closely (16 points per neighbour), in at most 62 dimensions
// (two columns of a 64-column operand block carry |x|^2 / 2).
bool filter_takes(uint64_t n, uint64_t d, uint64_t k);
// Whether it is faster than the full search for a group that it takes
// (FILTER_EUCLIDEAN, FILTER_COSINE; k counts the point itself), or for a batch:
// all its points, the largest k, and the cost of the group with the longest full
// search.
bool filter_pays(int mode, uint64_t n, uint64_t d, uint64_t k);
bool filter_pays_batched(uint64_t points, uint64_t d, uint64_t k, uint64_t group_cost);
// That search's time, in units of 10 ns.
inline uint64_t batched_group_cost(uint64_t n, uint64_t d, uint64_t k) {
    return n * (d <= 32 ? 5 : 9) + 160 * k;
}

struct FilterCall {
    const float* X;      // row-major rows, d floats each, any alignment
    uint64_t rows;       // rows in X
    int d;
    int mode;            // FILTER_*
    const float* norms;  // FILTER_COSINE: |x|^2 per row in the reference order
    std::vector<FilterSample> samples;  // base, out, n, k set; the groups the filter takes
    uint32_t* out_idx;
    float* out_dist;
    // queries the filter leaves to the full search, for every group:
    //   FILTER_BATCHED: a flag per block of redo_block queries, and the single
    //   queries while there are few
    //   else: query rows
    std::vector<uint32_t> ids;       // FILTER_BATCHED: the caller's id of each group
    std::vector<uint64_t> redo_off;  //   and the first flag of its blocks
    uint32_t redo_block;
    uint32_t* redo_flag;       // FILTER_BATCHED, device: redo_flags of them
    uint64_t redo_flags;
    uint2* redo_queries;       // FILTER_BATCHED, device: (group id, query), the first
    uint32_t* redo_queries_n;  // redo_short of redo_queries_n
    uint32_t redo_short;
    uint32_t* redo_rows;       // else, device: query rows and their number (zero before)
    uint32_t* redo_rows_n;
};

// Plans the call and uploads the plan (workspace from the context); `run`
// enqueues everything on a stream without waiting for the host or the GPU (so
// it can be captured).
struct FilterPlan {
    std::function<cudaError_t(cudaStream_t)> run;
    const float* Xt;  // not FILTER_BATCHED: column-major rows [d][rows], once `run` has run
};
FilterPlan filter_prepare(pq_ctx* c, FilterCall call);

}  // namespace pq
