// Exact brute-force kNN: neighbors::neighbors (crates/polariseq-core/src/
// neighbors.rs:101-147) bit for bit.
//
// For every query cell the reference scans all cells j = 0..n-1 in order,
// keeps a bounded max-heap of k_with_self = min(n_neighbors, n) entries
// (push with sift-up while short, else replace the root when d < root and
// sift down; neighbors.rs:160-212), stable-sorts it ascending, takes sqrt for
// Euclidean, and drops the first (closest) entry.  Distances use the
// reference's FP32 summation order (simd.rs): squared Euclidean, or cosine
// 1 - dot / (sqrt(|a|^2) sqrt(|b|^2)) (neighbors.rs:231-241).
//
// One warp per query, eight queries per CTA.  The CTA stages 32 candidate rows
// at a time in shared memory (16-byte padded rows, coalesced loads); lane j
// computes the distance to candidate j0 + j.  The heap update keeps the
// sequential semantics exactly: while the heap is short every candidate is
// pushed in order; after that a ballot finds the first lane (in j order) that
// beats the current root, lane 0 replaces and sifts, and the lanes before it
// are settled (the root only decreases, so a candidate that lost once loses
// again).  Cosine searches read per-row |x|^2 from a scratch array computed
// once (same summation order, so the values equal the reference's per-pair
// dot(b, b)).
//
// This full search is the form for d > 62, fewer than 16 points per
// neighbour, and callers without a workspace; otherwise the tensor-core filter
// (filter.cu) answers almost every query with the same bits, and k_redo_dist and
// k_redo_replay take those it leaves.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "exact.cuh"
#include "polariseq_knn.h"

namespace pq {
namespace {

constexpr int EW = 8;   // queries (warps) per CTA
constexpr int ET = 32;  // candidates per staged tile
constexpr uint32_t FULL = 0xFFFFFFFFu;

// Stage rows [r0, r0 + cnt) of the row-major n x d matrix into `dst` with
// row stride dp (zero padded).
__device__ __forceinline__ void stage_rows(const float* __restrict__ X, int d, int dp,
                                           uint64_t r0, uint32_t cnt, uint32_t rows,
                                           float* __restrict__ dst) {
    for (int t = threadIdx.x; t < int(rows) * dp; t += blockDim.x) {
        const int r = t / dp, c = t - r * dp;
        dst[t] = (uint32_t(r) < cnt && c < d) ? X[(r0 + r) * uint64_t(d) + c] : 0.0f;
    }
}

// |x|^2 of every row, dot(x, x) in the reference order (simd.rs:20-36:
// eight partial sums, ((a0+a4)+(a1+a5))+((a2+a6)+(a3+a7)), then the tail),
// with scalar loads (rows of the caller's matrix need not be 16-byte aligned).
__global__ void k_row_dots(const float* __restrict__ X, uint64_t n, int d,
                           float* __restrict__ norms) {
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* r = X + i * uint64_t(d);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int full = d >> 3;
    for (int c = 0; c < full; ++c)
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            const float v = r[8 * c + l];
            acc[l] = __fadd_rn(acc[l], __fmul_rn(v, v));
        }
    float tail = 0.0f;
    for (int j = full * 8; j < d; ++j) tail = __fadd_rn(tail, __fmul_rn(r[j], r[j]));
    const float s = __fadd_rn(__fadd_rn(__fadd_rn(acc[0], acc[4]), __fadd_rn(acc[1], acc[5])),
                              __fadd_rn(__fadd_rn(acc[2], acc[6]), __fadd_rn(acc[3], acc[7])));
    norms[i] = __fadd_rn(s, tail);
}

// Heap of one warp in shared memory (lane 0 mutates it), reference rules.
__device__ __forceinline__ void heap_push_up(float* hd, uint32_t* hi, int len, float d,
                                             uint32_t j) {
    int c = len;
    hd[c] = d;
    hi[c] = j;
    while (c > 0) {
        const int p = (c - 1) / 2;
        if (hd[c] > hd[p]) {
            const float tv = hd[c];
            hd[c] = hd[p];
            hd[p] = tv;
            const uint32_t ti = hi[c];
            hi[c] = hi[p];
            hi[p] = ti;
            c = p;
        } else {
            break;
        }
    }
}
// Both children are read at once and the new entry is written where it ends
// (the reference swaps it down level by level; the result is the same).
__device__ __forceinline__ void heap_replace_down(float* hd, uint32_t* hi, int len, float d,
                                                  uint32_t j) {
    int p = 0;
    for (;;) {
        const int l = 2 * p + 1, r = 2 * p + 2;
        const float dl = l < len ? hd[l] : d, dr = r < len ? hd[r] : d;
        int m = p;
        float dm = d;
        if (dl > dm) {
            m = l;
            dm = dl;
        }
        if (dr > dm) {
            m = r;
            dm = dr;
        }
        if (m == p) break;
        hd[p] = dm;
        hi[p] = hi[m];
        p = m;
    }
    hd[p] = d;
    hi[p] = j;
}

// The search's distance of rows a and b (16-byte aligned, zero padded); for the
// cosine metric an and bn are their |x|^2.
template <int D>
__device__ __forceinline__ float exact_dist(const float* __restrict__ a,
                                            const float* __restrict__ b, int d, int cosine,
                                            float an, float bn) {
    if (!cosine) return sq_dist_exact_t<D>(a, b, d);
    const float dt = dot_exact_t<D>(a, b, d);
    const float den = __fmul_rn(__fsqrt_rn(an), __fsqrt_rn(bn));
    return den > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(dt, den)) : 1.0f;
}

// One warp takes the distances dd of candidates j0 + lane (cnt of them) into
// its heap, as the reference's sequential scan does.
__device__ __forceinline__ void replay_tile(float* hd, uint32_t* hi, int& hlen, int kws, float dd,
                                            uint64_t j0, uint32_t cnt, int lane) {
    uint32_t pending = cnt == 32 ? FULL : ((1u << cnt) - 1u);
    // while the heap is short, every candidate is pushed in order
    while (pending && hlen < kws) {
        const int l = __ffs(pending) - 1;
        pending &= pending - 1;
        const float dl = __shfl_sync(FULL, dd, l);
        if (lane == 0) heap_push_up(hd, hi, hlen, dl, uint32_t(j0 + l));
        ++hlen;
        __syncwarp();
    }
    // then the first remaining lane that beats the current root, in order
    while (pending) {
        const float root = hd[0];
        const uint32_t m = __ballot_sync(FULL, ((pending >> lane) & 1u) && dd < root);
        if (!m) break;
        const int l = __ffs(m) - 1;
        pending &= ~((l == 31) ? FULL : ((2u << l) - 1u));
        const float dl = __shfl_sync(FULL, dd, l);
        if (lane == 0) heap_replace_down(hd, hi, hlen, dl, uint32_t(j0 + l));
        __syncwarp();
    }
}

// A warp's finished heap as the query's output row: stable ascending sort
// (insertion), sqrt for Euclidean, the closest entry dropped.
__device__ __forceinline__ void write_row(float* hd, uint32_t* hi, int hlen, int kws, uint64_t q,
                                          int cosine, int lane, uint32_t* __restrict__ out_idx,
                                          float* __restrict__ out_dist) {
    if (lane == 0) {
        for (int a = 1; a < hlen; ++a) {
            const float x = hd[a];
            const uint32_t y = hi[a];
            int b = a - 1;
            while (b >= 0 && hd[b] > x) {
                hd[b + 1] = hd[b];
                hi[b + 1] = hi[b];
                --b;
            }
            hd[b + 1] = x;
            hi[b + 1] = y;
        }
    }
    __syncwarp();
    const uint64_t per = uint64_t(kws - 1);
    for (int t = 1 + lane; t < hlen; t += 32) {
        out_idx[q * per + (t - 1)] = hi[t];
        out_dist[q * per + (t - 1)] = cosine ? hd[t] : __fsqrt_rn(hd[t]);
    }
}

template <int D>
__global__ void __launch_bounds__(EW * 32) k_exact_knn(const float* __restrict__ X, uint32_t n,
                                                       int d, int dp, int kws, int cosine,
                                                       const float* __restrict__ norms,
                                                       uint32_t* __restrict__ out_idx,
                                                       float* __restrict__ out_dist) {
    extern __shared__ __align__(16) float sm[];
    float* sq = sm;                 // EW x dp query rows
    float* st = sq + EW * dp;       // ET x dp candidate rows
    float* hd_all = st + ET * dp;   // EW x kws heap distances
    uint32_t* hi_all = reinterpret_cast<uint32_t*>(hd_all + EW * kws);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t q0 = uint64_t(blockIdx.x) * EW;
    const uint64_t q = q0 + w;
    const bool qv = q < n;
    stage_rows(X, d, dp, q0, uint32_t(n - q0 < EW ? n - q0 : EW), EW, sq);
    float* hd = hd_all + w * kws;
    uint32_t* hi = hi_all + w * kws;
    const float* qr = sq + w * dp;
    const float qn = (cosine && qv) ? norms[q] : 0.0f;
    int hlen = 0;  // warp-uniform
    for (uint64_t j0 = 0; j0 < n; j0 += ET) {
        const uint32_t cnt = uint32_t(n - j0 < ET ? n - j0 : ET);
        __syncthreads();  // the previous tile is consumed
        stage_rows(X, d, dp, j0, cnt, ET, st);
        __syncthreads();
        if (!qv) continue;
        float dd = 0.0f;
        if (uint32_t(lane) < cnt)
            dd = exact_dist<D>(qr, st + lane * dp, d, cosine, qn, cosine ? norms[j0 + lane] : 0.0f);
        replay_tile(hd, hi, hlen, kws, dd, j0, cnt, lane);
    }
    if (qv) write_row(hd, hi, hlen, kws, q, cosine, lane, out_idx, out_dist);
}

// Single queries (those the filter leaves: equal distances among the k + 1
// nearest, whose order is the heap's), in two steps: k_redo_dist evaluates all
// their distances, and k_redo_replay walks them as the sequential scan does, a
// warp per query.  A CTA per query that did both waited for row loads between
// barriers (346 us for 17 queries at 20,000 x 50, 4.6 ms for 2,762 at 60,013 x
// 30 cosine).  The distance buffer holds redo_cap queries; k_redo_rest takes
// those past them.
constexpr int RQ = int(EXACT_REDO_Q);  // queries per CTA of k_redo_dist
constexpr int RD = 256;                // candidates (= threads) per CTA

// dist[u * ld] of RQ queries (their rows in sq, dimension-major) and row j;
// rows are column-major, so every load is one coalesced line.
template <int D>
__device__ __forceinline__ void redo_dist4(const float* __restrict__ Xt, uint32_t n, int d_,
                                           int cosine, const float* __restrict__ norms,
                                           const float (*sq)[RQ], const float* qn, uint32_t j,
                                           uint32_t ld, float* __restrict__ dist) {
    const int d = D > 0 ? D : d_, full = d >> 3;
    const float* col = Xt + j;
    float acc[RQ][8], tail[RQ];
#pragma unroll
    for (int u = 0; u < RQ; ++u) {
        tail[u] = 0.0f;
#pragma unroll
        for (int l = 0; l < 8; ++l) acc[u][l] = 0.0f;
    }
    auto term = [&](float a, float x, float y) {
        const float t = cosine ? x : __fsub_rn(x, y);
        return __fadd_rn(a, __fmul_rn(t, cosine ? y : t));
    };
#pragma unroll 2
    for (int c = 0; c < full; ++c) {
        float y[8];
#pragma unroll
        for (int l = 0; l < 8; ++l) y[l] = col[size_t(8 * c + l) * n];
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            const float4 x = *reinterpret_cast<const float4*>(sq[8 * c + l]);
            acc[0][l] = term(acc[0][l], x.x, y[l]);
            acc[1][l] = term(acc[1][l], x.y, y[l]);
            acc[2][l] = term(acc[2][l], x.z, y[l]);
            acc[3][l] = term(acc[3][l], x.w, y[l]);
        }
    }
    for (int c = 8 * full; c < d; ++c) {
        const float y = col[size_t(c) * n];
#pragma unroll
        for (int u = 0; u < RQ; ++u) tail[u] = term(tail[u], sq[c][u], y);
    }
#pragma unroll
    for (int u = 0; u < RQ; ++u) {
        const float* A = acc[u];
        float r = __fadd_rn(
            __fadd_rn(__fadd_rn(__fadd_rn(A[0], A[4]), __fadd_rn(A[1], A[5])),
                      __fadd_rn(__fadd_rn(A[2], A[6]), __fadd_rn(A[3], A[7]))),
            tail[u]);
        if (cosine) {
            const float den = __fmul_rn(__fsqrt_rn(qn[u]), __fsqrt_rn(norms[j]));
            r = den > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(r, den)) : 1.0f;
        }
        dist[size_t(u) * ld] = r;
    }
}

// The rows of queries [i0, i0 + RQ) of the list (the last one repeated past its
// end).
__device__ __forceinline__ void redo_queries(const float* __restrict__ Xt, uint32_t n, int d,
                                             int cosine, const float* __restrict__ norms,
                                             const uint32_t* __restrict__ list, uint32_t nq,
                                             uint32_t i0, float (*sq)[RQ], float* qn) {
    for (int t = threadIdx.x; t < d * RQ; t += blockDim.x)
        sq[t / RQ][t % RQ] = Xt[size_t(t / RQ) * n + list[min(i0 + uint32_t(t % RQ), nq - 1)]];
    if (threadIdx.x < RQ)
        qn[threadIdx.x] = cosine ? norms[list[min(i0 + threadIdx.x, nq - 1)]] : 0.0f;
}

// One warp: the sequential scan over a query's distances to candidates [c0, c0 +
// n) (512 in flight, 128 per vote).
__device__ __forceinline__ void redo_scan(const float* __restrict__ row, uint32_t c0, uint32_t n,
                                          int kws, float* hd, uint32_t* hi, int& hlen) {
    const int lane = threadIdx.x & 31;
    for (uint32_t j0 = 0; j0 < n; j0 += 512) {
        float dd[16];
#pragma unroll
        for (int g = 0; g < 16; ++g) {
            const uint32_t j = j0 + 32 * g + lane;
            dd[g] = j < n ? row[j] : __int_as_float(0x7f800000);
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            bool hit = hlen < kws;
#pragma unroll
            for (int g = 4 * v; g < 4 * v + 4; ++g) hit |= hlen == kws && dd[g] < hd[0];
            if (!__any_sync(FULL, hit)) continue;
#pragma unroll
            for (int g = 4 * v; g < 4 * v + 4; ++g) {
                const uint32_t jg = j0 + 32 * g;
                if (jg < n)
                    replay_tile(hd, hi, hlen, kws, dd[g], c0 + jg, n - jg < 32 ? n - jg : 32, lane);
            }
        }
    }
}

// The first cap queries of the list: distances over the whole grid ...
template <int D>
__global__ void __launch_bounds__(RD) k_redo_dist(const float* __restrict__ Xt, uint32_t n, int d,
                                                  int cosine, const float* __restrict__ norms,
                                                  const uint32_t* __restrict__ list,
                                                  const uint32_t* __restrict__ list_n,
                                                  uint32_t cap, uint32_t ld,
                                                  float* __restrict__ dist) {
    __shared__ __align__(16) float sq[64][RQ];
    __shared__ float qn[RQ];
    const uint32_t nq = min(*list_n, cap), j = blockIdx.x * RD + threadIdx.x;
    for (uint32_t i0 = blockIdx.y * RQ; i0 < nq; i0 += gridDim.y * RQ) {
        __syncthreads();
        redo_queries(Xt, n, d, cosine, norms, list, nq, i0, sq, qn);
        __syncthreads();
        if (j < n)
            redo_dist4<D>(Xt, n, d, cosine, norms, sq, qn, j, ld, dist + size_t(i0) * ld + j);
    }
}
// ... and their scans, a warp each.
__global__ void __launch_bounds__(32) k_redo_replay(const float* __restrict__ dist, uint32_t n,
                                                    uint32_t ld, int kws, int cosine,
                                                    const uint32_t* __restrict__ list,
                                                    const uint32_t* __restrict__ list_n,
                                                    uint32_t cap, uint32_t* __restrict__ out_idx,
                                                    float* __restrict__ out_dist) {
    __shared__ float hd[EXACT_MAX_K];
    __shared__ uint32_t hi[EXACT_MAX_K];
    const uint32_t nq = min(*list_n, cap);
    for (uint32_t i = blockIdx.x; i < nq; i += gridDim.x) {
        int hlen = 0;
        redo_scan(dist + size_t(i) * ld, 0, n, kws, hd, hi, hlen);
        write_row(hd, hi, hlen, kws, list[i], cosine, threadIdx.x, out_idx, out_dist);
        __syncwarp();
    }
}
// The queries past the first cap (inputs full of ties, or that the filter's
// bounds do not cover): RQ per CTA at a time, `seg` candidates after another
// through the CTA's own part of the buffer, so that the grid fills the chip
// whatever the number of points.  (With whole rows per CTA the buffer held 134
// CTAs at 500,000 points.)
template <int D>
__global__ void __launch_bounds__(RD) k_redo_rest(const float* __restrict__ Xt, uint32_t n, int d,
                                                  int kws, int cosine,
                                                  const float* __restrict__ norms,
                                                  const uint32_t* __restrict__ list,
                                                  const uint32_t* __restrict__ list_n,
                                                  uint32_t cap, uint32_t seg,
                                                  float* __restrict__ dist,
                                                  uint32_t* __restrict__ out_idx,
                                                  float* __restrict__ out_dist) {
    __shared__ __align__(16) float sq[64][RQ];
    __shared__ float qn[RQ];
    __shared__ float hd[RQ][EXACT_MAX_K];
    __shared__ uint32_t hi[RQ][EXACT_MAX_K];
    const uint32_t nq = *list_n, w = threadIdx.x >> 5;
    float* mine = dist + size_t(blockIdx.x) * RQ * seg;
    for (uint32_t i0 = cap + blockIdx.x * RQ; i0 < nq; i0 += gridDim.x * RQ) {
        __syncthreads();
        redo_queries(Xt, n, d, cosine, norms, list, nq, i0, sq, qn);
        const bool scans = w < uint32_t(RQ) && i0 + w < nq;
        int hlen = 0;
        for (uint32_t c0 = 0; c0 < n; c0 += seg) {
            const uint32_t len = min(seg, n - c0);
            __syncthreads();  // the queries are there, the last segment is scanned
            for (uint32_t j = threadIdx.x; j < len; j += RD)
                redo_dist4<D>(Xt, n, d, cosine, norms, sq, qn, c0 + j, seg, mine + j);
            __syncthreads();
            if (scans) redo_scan(mine + size_t(w) * seg, c0, len, kws, hd[w], hi[w], hlen);
        }
        if (scans)
            write_row(hd[w], hi[w], hlen, kws, list[i0 + w], cosine, threadIdx.x & 31, out_idx,
                      out_dist);
    }
}

__global__ void k_exact_indptr(uint32_t* __restrict__ indptr, uint64_t n, uint32_t per) {
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i <= n) indptr[i] = uint32_t(i * per);
}

template <int D>
cudaError_t launch_d(const float* X, uint64_t n, int d, int kws, int cosine, float* norms,
                     uint32_t* indptr, uint32_t* indices, float* dists, cudaStream_t st,
                     const ExactFilter* filter) {
    const int dp = (d + 3) / 4 * 4;
    if (cosine) {
        k_row_dots<<<uint32_t((n + 255) / 256), 256, 0, st>>>(X, n, d, norms);
        count_launch();
    }
    if (filter) {
        cudaError_t e = cudaMemsetAsync(filter->redo_n, 0, 4, st);
        if (e == cudaSuccess) e = filter->run(st);
        if (e != cudaSuccess) return e;
        const uint32_t cap = filter->redo_cap, ld = filter->redo_ld;
        const dim3 grid(uint32_t((n + RD - 1) / RD), 16);
        k_redo_dist<D><<<grid, RD, 0, st>>>(filter->Xt, uint32_t(n), d, cosine, norms, filter->redo,
                                            filter->redo_n, cap, ld, filter->redo_dist);
        k_redo_replay<<<148 * 16, 32, 0, st>>>(filter->redo_dist, uint32_t(n), ld, kws, cosine,
                                              filter->redo, filter->redo_n, cap, indices, dists);
        k_redo_rest<D><<<EXACT_REDO_CTAS, RD, 0, st>>>(
            filter->Xt, uint32_t(n), d, kws, cosine, norms, filter->redo, filter->redo_n, cap,
            exact_redo_seg(ld), filter->redo_dist, indices, dists);
        count_launch();
        count_launch();
        count_launch();
    } else {
        k_exact_knn<D><<<uint32_t((n + EW - 1) / EW), EW * 32, exact_knn_smem(d, kws), st>>>(
            X, uint32_t(n), d, dp, kws, cosine, norms, indices, dists);
        count_launch();
    }
    k_exact_indptr<<<uint32_t((n + 256) / 256), 256, 0, st>>>(indptr, n, uint32_t(kws - 1));
    count_launch();
    return cudaGetLastError();
}

}  // namespace

size_t exact_knn_smem(int d, int kws) {
    const int dp = (d + 3) / 4 * 4;
    return size_t(EW + ET) * dp * 4 + size_t(EW) * kws * 8;
}

cudaError_t exact_knn_prepare() {
    cudaFuncAttributes fa;
    cudaError_t e;
    if ((e = cudaFuncGetAttributes(&fa, k_row_dots)) != cudaSuccess) return e;
    if ((e = cudaFuncGetAttributes(&fa, k_exact_indptr)) != cudaSuccess) return e;
    const int smax = int(exact_knn_smem(EXACT_MAX_DIM, EXACT_MAX_K));
    if ((e = cudaFuncSetAttribute(k_exact_knn<50>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  smax)) != cudaSuccess)
        return e;
    return cudaFuncSetAttribute(k_exact_knn<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax);
}

cudaError_t launch_exact_knn(const float* X, uint64_t n, int d, int kws, int cosine,
                             float* norms, uint32_t* indptr, uint32_t* indices, float* dists,
                             cudaStream_t st, const ExactFilter* filter) {
    if (n == 0 || n > 0xFFFFFFFEull || d < 1 || d > EXACT_MAX_DIM || kws < 1 ||
        kws > EXACT_MAX_K)
        return cudaErrorInvalidValue;
    if (d == 50)
        return launch_d<50>(X, n, d, kws, cosine, norms, indptr, indices, dists, st, filter);
    return launch_d<0>(X, n, d, kws, cosine, norms, indptr, indices, dists, st, filter);
}

}  // namespace pq

// ── allocation-free variant ─────────────────────────────────────────────────
// Scratch of pq_neighbors_into_device_noalloc: the cosine metric's per-row
// |x|^2, for at most EXACT_NOALLOC_MAX_ROWS rows (1 MiB).  It lives in every
// device that loads the library, from load until process exit.  In host code
// the name below stands for a host-side shadow, not the device array: the
// device address comes from cudaGetSymbolAddress at set-up.
namespace pq {
namespace {

constexpr uint64_t EXACT_NOALLOC_MAX_ROWS = uint64_t(1) << 18;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) float g_noalloc_norms[EXACT_NOALLOC_MAX_ROWS];

std::mutex g_noalloc_mu;
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};

// Once per device, with that device current: the scratch array's device
// address, and the kernels loaded with their shared-memory limit raised.
cudaError_t noalloc_setup(int dev, float** out) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        float* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_noalloc_norms);
        if (e != cudaSuccess) return e;
        if ((e = exact_knn_prepare()) != cudaSuccess) return e;
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

}  // namespace
}  // namespace pq

extern "C" int pq_neighbors_into_device_noalloc(const float* d_data, uint64_t n_obs,
                                                uint64_t n_dim, uint64_t n_neighbors,
                                                int32_t metric, uint32_t* d_indptr,
                                                uint32_t* d_indices, float* d_dists,
                                                uint64_t* nnz_out, void* stream) {
    using namespace pq;
    if (!d_data || !d_indptr || !d_indices || !d_dists || !nnz_out) return PQ_EINVAL;
    if (n_obs == 0 || n_dim == 0 || n_neighbors == 0) return PQ_EINVAL;
    if (metric != PQ_METRIC_EUCLIDEAN && metric != PQ_METRIC_COSINE) return PQ_EINVAL;
    if (n_obs > EXACT_NOALLOC_MAX_ROWS) return PQ_ETOOBIG;
    const uint64_t kws = n_neighbors < n_obs ? n_neighbors : n_obs;
    if (kws > uint64_t(EXACT_MAX_K) || n_dim > uint64_t(EXACT_MAX_DIM)) return PQ_ENOTSUP;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        cudaGetLastError();
        return PQ_EDEVICE;
    }
    float* norms = nullptr;
    if (noalloc_setup(dev, &norms) != cudaSuccess) {
        cudaGetLastError();
        return PQ_EDEVICE;
    }
    // every norm the search reads is written first, on the same stream
    if (launch_exact_knn(d_data, n_obs, int(n_dim), int(kws), metric == PQ_METRIC_COSINE, norms,
                         d_indptr, d_indices, d_dists,
                         static_cast<cudaStream_t>(stream)) != cudaSuccess) {
        cudaGetLastError();
        return PQ_EDEVICE;
    }
    *nnz_out = n_obs * (kws - 1);
    return PQ_OK;
}
