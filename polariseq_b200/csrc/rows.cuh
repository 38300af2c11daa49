// Whole-row staging of gathered embedding rows in shared memory, per warp.
//
// A thread that reads its own row 16 bytes at a time makes every load of its
// warp touch 32 lines, and such gathers were bound by those wavefronts: 13 per
// 52-float row and point, one per cycle (the forest's margins measured 11-13
// cycles per point on one SM).  Here 8 or 16 lanes copy one row
// (asynchronously, past the registers), so a load instruction touches 2-5
// lines, and every lane then reads its own row from shared memory.  Rows sit
// an odd number of 16-byte units apart, so that neighbouring rows start in
// different banks.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "seq_plan.cuh"

namespace pq {

// 16-byte asynchronous global -> shared copy (both addresses 16-byte aligned),
// bypassing L1.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The converged warp starts the copies of rows X[id of lane r], r < cnt, to
// dst + r * rs.
__device__ __forceinline__ void warp_stage_rows(const float* __restrict__ X, int dp, int rs,
                                                uint32_t id, uint32_t cnt, float* dst) {
    const int lane = threadIdx.x & 31, q4 = dp / 4;
    if (q4 <= 8) {
        const int rr0 = lane >> 3, cc = lane & 7;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int rr = u * 4 + rr0;
            const uint32_t j = __shfl_sync(0xFFFFFFFFu, id, rr);
            if (cc < q4 && uint32_t(rr) < cnt)
                cp_async16(dst + rr * rs + cc * 4, X + size_t(j) * dp + cc * 4);
        }
    } else if (q4 <= 16) {
        const int rr0 = lane >> 4, cc = lane & 15;
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            const int rr = u * 2 + rr0;
            const uint32_t j = __shfl_sync(0xFFFFFFFFu, id, rr);
            if (cc < q4 && uint32_t(rr) < cnt)
                cp_async16(dst + rr * rs + cc * 4, X + size_t(j) * dp + cc * 4);
        }
    } else {
        for (uint32_t rr = 0; rr < cnt; ++rr) {
            const uint32_t j = __shfl_sync(0xFFFFFFFFu, id, int(rr));
            for (int cc = lane; cc < q4; cc += 32)
                cp_async16(dst + rr * rs + cc * 4, X + size_t(j) * dp + cc * 4);
        }
    }
}

}  // namespace pq
