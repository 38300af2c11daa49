// Shared-memory plan of the RP subtree kernel (subtree.cu) and of staged rows
// (rows.cuh).  No CUDA types: a host compiler can check it too.
#pragma once

#include <stddef.h>
#include <stdint.h>

#ifndef PQ_PLAN
#ifdef __CUDACC__
#define PQ_PLAN __host__ __device__ __forceinline__
#else
#define PQ_PLAN inline
#endif
#endif

namespace pq {

// Shared memory a CTA may have (227 KB), static arrays included.
constexpr size_t SMEM_PER_CTA = 232448;
// A kernel's limit on dynamic shared memory belongs to the device, not to a
// context: every launch sets the same limit, whatever it needs itself, so that
// contexts on several threads do not lower each other's between setting and
// launching.  (For kernels with less than 2 KB of static arrays.)
constexpr int SMEM_DYNAMIC = int(SMEM_PER_CTA) - 2048;

// Floats between staged rows of dp floats (dp a multiple of 4).
PQ_PLAN int staged_stride(int dp) { return (dp / 4) % 2 ? dp : dp + 4; }

// Dynamic shared memory of a subtree CTA with `rows` staged rows: the normal
// and the offset's terms (dp floats each), then the rows.
PQ_PLAN size_t seq_dynamic(int dp, int rows) {
    return size_t(2 * dp) * 4 + size_t(rows) * size_t(staged_stride(dp)) * 4;
}
// Staged rows: at most `cap`, in at most `room` bytes, and beside what the CTA
// has already (`fixed` bytes of static arrays, and the two vectors).
PQ_PLAN int seq_staged_rows(int dp, int cap, size_t room, size_t fixed) {
    const size_t row = size_t(staged_stride(dp)) * 4, taken = fixed + seq_dynamic(dp, 0);
    const size_t left = taken < SMEM_PER_CTA ? SMEM_PER_CTA - taken : 0;
    const size_t fit = (left < room ? left : room) / row;
    const int rows = fit < size_t(cap) ? int(fit) : cap;
    return rows < 2 ? 0 : rows;
}

}  // namespace pq
