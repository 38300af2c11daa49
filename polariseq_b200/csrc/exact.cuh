// Exact brute-force kNN (neighbors::neighbors) launch interface.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <functional>

namespace pq {

constexpr int EXACT_MAX_DIM = 512;  // n_dim limit of the staged-tile kernel
constexpr int EXACT_MAX_K = 256;    // k_with_self limit (per-warp shared-memory heap)

size_t exact_knn_smem(int d, int kws);
// Loads the kernels and raises their shared-memory limit on the current
// device (once per device, before the first launch).
cudaError_t exact_knn_prepare();
// Enqueues the search on `st`: indptr (n+1), indices / dists (n * (kws-1)).
// `norms` (n floats) is scratch for the cosine metric (unused for Euclidean);
// every element the kernels read is written first in the same launch sequence.
// With `filter`, its prepared steps run first (after the norms) and the search
// takes the queries they leave in `redo`.
struct ExactFilter {
    std::function<cudaError_t(cudaStream_t)> run;
    uint32_t* redo;    // device: query rows
    uint32_t* redo_n;  // device: their number
    const float* Xt;   // device: the rows column-major [d][n], written by `run`
    float* redo_dist;  // device: distances of redo_cap queries, redo_ld apart; at least
                       // exact_redo_floats(redo_ld) floats for the queries past them
    uint32_t redo_cap, redo_ld;
};
constexpr uint32_t EXACT_REDO_Q = 4;          // queries at a time per CTA
constexpr uint32_t EXACT_REDO_CTAS = 148 * 4;
// Their candidates at a time: whole rows while those of every CTA fit in 620 MB,
// else 8,192.  (Segments of 8,192 at 60,000 points: 48.6 -> 44.8 ms with a zero
// row at k = 15, but 19.6 -> 20.1 with ties at k = 100, where the scans' barriers
// count; at 200,000 points 727 -> 475.)
inline uint32_t exact_redo_seg(uint32_t ld) { return ld <= 65536 ? ld : 8192; }
inline size_t exact_redo_floats(uint32_t ld) {
    return size_t(EXACT_REDO_CTAS) * EXACT_REDO_Q * exact_redo_seg(ld);
}
cudaError_t launch_exact_knn(const float* X, uint64_t n, int d, int kws, int cosine,
                             float* norms, uint32_t* indptr, uint32_t* indices, float* dists,
                             cudaStream_t st, const ExactFilter* filter = nullptr);

}  // namespace pq
