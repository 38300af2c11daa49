// RP-tree forest of the plain form, bit-exact with the reference's
// build_tree (crates/polariseq-core/src/nndescent.rs:356-646).
//
// Top levels (rp_tree_parallel, :587-641: nodes of >= 8192 points above depth
// 6) are processed level by level for all trees at once: one hyperplane per
// node, one thread per (tree, position) for the margins, and a closed-form
// parallel restatement of the two-pointer partition (:389-405).  Below that
// every subtree is finished by one CTA in depth-first order (subtree.cu).
//
// The two-pointer partition moves, for a node with nL left points:
//   left  point at p <  nL          -> p
//   right point at p <  nL, rank j  -> (j == 1 ? size : B[j-1]) - 1
//   left  point at p >= nL, rank j  -> A[j]          (rank from the top)
//   right point at p >  nL          -> p - 1
//   right point at p == nL          -> (c == 0 ? size : B[c]) - 1
// where A[j] is the position of the j-th right point in [0, nL), B[j] the
// position of the j-th left point in [nL, size) counted from the top, and c
// the number of right points in [0, nL).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "primitives.cuh"
#include "rows.cuh"

namespace pq {
namespace {

constexpr int FT = 256;             // threads per forest CTA
constexpr int PER = FOREST_CHUNK / FT;  // positions per thread in a chunk

// Exclusive block scan of one u32 per thread (any multiple of 32 threads, at
// most 1024); *total receives the block sum.
__device__ __forceinline__ uint32_t bscan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t s = lane < nw ? ws[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) ws[lane] = s;
    }
    __syncthreads();
    uint32_t r = (w > 0 ? ws[w - 1] : 0) + x - v;
    *total = ws[nw - 1];
    __syncthreads();
    return r;
}

// random_hyperplane (nndescent.rs:367-385) for one top-level node.
__global__ void k_hyper(ForestArgs a, PNode* nodes, float* normals) {
    __shared__ uint32_t sA, sB;
    PNode nd = nodes[blockIdx.x];
    if (threadIdx.x == 0) {
        Rng r{nd.seed};
        const uint32_t* ids = a.ids + size_t(nd.tree) * a.n + nd.start;
        uint32_t A = ids[r.below(nd.size)];
        uint32_t B = ids[r.below(nd.size)];
        int tries = 0;
        while (B == A && tries < 8) {
            B = ids[r.below(nd.size)];
            ++tries;
        }
        sA = A;
        sB = B;
        nodes[blockIdx.x].rng_after = r.s;
    }
    __syncthreads();
    const float* xa = a.X + size_t(sA) * a.dp;
    const float* xb = a.X + size_t(sB) * a.dp;
    float* nv = normals + size_t(blockIdx.x) * a.dp;
    for (int j = threadIdx.x; j < a.dp; j += blockDim.x)
        nv[j] = j < a.d ? __fsub_rn(xa[j], xb[j]) : 0.0f;
    if (threadIdx.x == 0) {
        float s = -0.0f;  // Rust's f32 sum folds from -0.0
        for (int j = 0; j < a.d; ++j) {
            float nvj = __fsub_rn(xa[j], xb[j]);
            s = __fadd_rn(s, __fmul_rn(__fmul_rn(nvj, 0.5f), __fadd_rn(xa[j], xb[j])));
        }
        nodes[blockIdx.x].offset = -s;
    }
}

// Margins of a top-level chunk; ties go by splitmix(seed ^ id) & 1 (:599-607).
// Rows are staged 32 per warp (rows.cuh) when they fit (staged = their stride,
// else 0: a thread reads its own row).
__global__ void __launch_bounds__(FT) k_sides(ForestArgs a, const PNode* nodes,
                                              const uint32_t* chunk_node, const float* normals,
                                              uint32_t* chunkL, int staged) {
    extern __shared__ __align__(16) float nv[];
    __shared__ uint32_t ws[32];
    const uint32_t ni = chunk_node[blockIdx.x];
    const PNode nd = nodes[ni];
    for (int j = threadIdx.x; j < a.dp; j += FT) nv[j] = normals[size_t(ni) * a.dp + j];
    __syncthreads();
    const uint32_t off = (blockIdx.x - nd.chunk0) * FOREST_CHUNK;
    const uint32_t len = min(uint32_t(FOREST_CHUNK), nd.size - off);
    const size_t tb = size_t(nd.tree) * a.n + nd.start + off;
    const uint32_t lane = threadIdx.x & 31, w0 = threadIdx.x - lane;
    float* rows = nv + a.dp + size_t(w0) * staged;
    uint32_t cnt = 0;
    uint32_t id = w0 < len ? a.ids[tb + min(w0 + lane, len - 1)] : 0u;
    for (uint32_t i0 = w0; i0 < len; i0 += FT) {
        const uint32_t i = i0 + lane;
        const float* x = a.X + size_t(id) * a.dp;
        const uint32_t cur = id;
        if (staged) {
            warp_stage_rows(a.X, a.dp, staged, id, min(32u, len - i0), rows);
            cp_async_commit();
            x = rows + lane * staged;
        }
        if (i0 + FT < len) id = a.ids[tb + min(i + FT, len - 1)];  // the next rows' ids
        if (staged) {
            cp_async_wait<0>();
            __syncwarp();
        }
        if (i < len) {
            const float m = __fadd_rn(dot_exact(nv, x, a.d), nd.offset);
            const bool left = fabsf(m) < 1e-8f ? ((splitmix(nd.seed ^ uint64_t(cur)) & 1ull) == 0)
                                               : (m > 0.0f);
            a.side[tb + i] = left ? 1 : 0;
            cnt += left;
        }
        __syncwarp();
    }
    uint32_t tot;
    bscan(cnt, ws, &tot);
    if (threadIdx.x == 0) chunkL[blockIdx.x] = tot;
}

// Per node: exclusive prefix of its chunks' left counts; nL = total.
__global__ void k_node_scan(PNode* nodes, uint32_t nn, uint32_t* chunkL) {
    uint32_t ni = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (ni >= nn) return;
    const int lane = threadIdx.x & 31;
    PNode nd = nodes[ni];
    uint32_t nch = (nd.size + FOREST_CHUNK - 1) / FOREST_CHUNK;
    uint32_t run = 0;
    for (uint32_t b = 0; b < nch; b += 32) {
        uint32_t c = b + lane;
        uint32_t v = c < nch ? chunkL[nd.chunk0 + c] : 0;
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        if (c < nch) chunkL[nd.chunk0 + c] = run + x - v;
        run += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (lane == 0) {
        nodes[ni].nL = run;
        nodes[ni].c = 0;
    }
}

// Pass 1 of the partition: rank tables A/B and c (see the file comment).
__global__ void __launch_bounds__(FT) k_part_tables(ForestArgs a, PNode* nodes,
                                                    const uint32_t* chunk_node,
                                                    const uint32_t* chunkPre) {
    __shared__ uint32_t ws[32];
    const uint32_t ni = chunk_node[blockIdx.x];
    const PNode nd = nodes[ni];
    const uint32_t off = (blockIdx.x - nd.chunk0) * FOREST_CHUNK;
    const uint32_t len = min(uint32_t(FOREST_CHUNK), nd.size - off);
    const size_t nb = size_t(nd.tree) * a.n + nd.start;
    uint8_t s[PER];
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        uint32_t i = threadIdx.x * PER + j;
        s[j] = i < len ? a.side[nb + off + i] : 0;
        cnt += s[j];
    }
    uint32_t tot;
    uint32_t lp = chunkPre[blockIdx.x] + bscan(cnt, ws, &tot);
    const uint32_t nL = nd.nL;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        uint32_t i = threadIdx.x * PER + j;
        if (i < len) {
            uint32_t p = off + i;
            if (s[j]) {
                if (p >= nL) a.tabB[nb + (nL - lp) - 1] = p;
            } else {
                if (p < nL) a.tabA[nb + (p - lp)] = p;  // rank p-lp+1, 0-based p-lp
            }
            if (p == nL) nodes[ni].c = nL - lp;
            lp += s[j];
        }
    }
}

// Pass 2: scatter ids to their partitioned positions in tmp.
__global__ void __launch_bounds__(FT) k_part_scatter(ForestArgs a, const PNode* nodes,
                                                     const uint32_t* chunk_node,
                                                     const uint32_t* chunkPre) {
    __shared__ uint32_t ws[32];
    const uint32_t ni = chunk_node[blockIdx.x];
    const PNode nd = nodes[ni];
    const uint32_t off = (blockIdx.x - nd.chunk0) * FOREST_CHUNK;
    const uint32_t len = min(uint32_t(FOREST_CHUNK), nd.size - off);
    const size_t nb = size_t(nd.tree) * a.n + nd.start;
    uint8_t s[PER];
    uint32_t cnt = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        uint32_t i = threadIdx.x * PER + j;
        s[j] = i < len ? a.side[nb + off + i] : 0;
        cnt += s[j];
    }
    uint32_t tot;
    uint32_t lp = chunkPre[blockIdx.x] + bscan(cnt, ws, &tot);
    const uint32_t nL = nd.nL, size = nd.size, c = nd.c;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        uint32_t i = threadIdx.x * PER + j;
        if (i < len) {
            uint32_t p = off + i, dst;
            if (s[j]) {
                dst = p < nL ? p : a.tabA[nb + (nL - lp) - 1];
            } else if (p < nL) {
                uint32_t r = p - lp + 1;
                dst = (r == 1 ? size : a.tabB[nb + r - 2]) - 1;
            } else if (p > nL) {
                dst = p - 1;
            } else {
                dst = (c == 0 ? size : a.tabB[nb + c - 1]) - 1;
            }
            a.tmp[nb + dst] = a.ids[nb + p];
            lp += s[j];
        }
    }
}

__global__ void __launch_bounds__(FT) k_part_copy(ForestArgs a, const PNode* nodes,
                                                  const uint32_t* chunk_node) {
    const uint32_t ni = chunk_node[blockIdx.x];
    const PNode nd = nodes[ni];
    const uint32_t off = (blockIdx.x - nd.chunk0) * FOREST_CHUNK;
    const uint32_t len = min(uint32_t(FOREST_CHUNK), nd.size - off);
    const size_t nb = size_t(nd.tree) * a.n + nd.start + off;
    for (uint32_t i = threadIdx.x; i < len; i += FT) a.ids[nb + i] = a.tmp[nb + i];
}

// random_split (nndescent.rs:408-415) where the hyperplane separated nothing.
__global__ void k_degenerate(ForestArgs a, PNode* nodes, uint32_t nn) {
    uint32_t ni = blockIdx.x * blockDim.x + threadIdx.x;
    if (ni >= nn) return;
    PNode nd = nodes[ni];
    if (nd.nL != 0 && nd.nL != nd.size) return;
    Rng r{nd.rng_after};
    uint32_t* ids = a.ids + size_t(nd.tree) * a.n + nd.start;
    for (uint32_t i = nd.size - 1; i >= 1; --i) {
        uint32_t j = uint32_t(r.below(uint64_t(i) + 1));
        uint32_t t = ids[i];
        ids[i] = ids[j];
        ids[j] = t;
    }
    nodes[ni].nL = nd.size / 2;
}

// Leaf starts of all trees: flags (u8) -> u32 -> one exclusive scan over the
// trees' positions -> each tree's positions from its own first leaf.  One pass
// for all trees instead of five launches per tree (48 trees at 20,000 cells:
// 240 launches of a few microseconds).
__global__ void k_flags_u32(const uint8_t* f, size_t tn, uint32_t* out) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < tn) out[i] = f[i];
}
__global__ void k_leaf_scatter(const uint8_t* f, const uint32_t* pre, size_t tn, uint32_t n,
                               uint32_t* leaf_start) {
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= tn || !f[i]) return;
    const size_t t0 = i / n * n;
    leaf_start[t0 + (pre[i] - pre[t0])] = uint32_t(i - t0);
}
__global__ void k_leaf_counts(const uint32_t* pre, const uint64_t* total, uint32_t T, uint32_t n,
                              uint64_t* counts) {
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const uint64_t end = t + 1 < T ? uint64_t(pre[size_t(t + 1) * n]) : *total;
    counts[t] = end - pre[size_t(t) * n];
}

// Leaf all-pairs of one tree (nndescent.rs:785-815).  The member at a
// position receives every other member of its leaf in leaf order, which is
// the order the reference's (i<j, p-then-q) generation addresses it.
//
// A CTA takes lpb consecutive leaves (as many as fit LCAP positions at the
// tree's leaf size, at most LPB): it stages their ids, rows and their
// members' heap rows in shared memory once (the heap rows column-major, one
// column per position, so that the pushes of a warp hit distinct banks),
// computes each pair's distance once into a per-position table, and then each
// thread replays its own member's pushes on the staged row; the changed rows
// go back.  The heap rows move between global and shared memory in position x
// slot order (consecutive threads on one row's slots: coalesced), the staged
// columns LCAP + 1 apart so that those accesses spread over the banks.  A push whose distance is not below the row's root (its
// current worst) is rejected unchanged (nndescent.rs:176).  Tiles whose span
// exceeds LCAP or whose leaves exceed LMAX members take the direct path.
constexpr int LPB = 8;      // leaves per CTA, at most
constexpr int LCAP = 128;   // staged positions per CTA (= threads)
constexpr int LMAXC = 64;   // largest leaf of the staged path
constexpr int HS = LCAP + 1;  // column stride of the staged heap rows

size_t leaf_pairs_smem(int dp, int lmax, int k) {
    return size_t(LCAP) * dp * 4 + size_t(LCAP) * lmax * 4 + size_t(HS) * k * 9;
}

template <int D>
__global__ void __launch_bounds__(LCAP) k_leaf_pairs(
    const float* __restrict__ X, int d, int dp, const uint32_t* __restrict__ ids,
    const uint32_t* __restrict__ leaf_start, uint32_t nleaves, uint32_t n, int k, uint32_t* hidx,
    float* hdist, uint8_t* hflag, int LMAX, int lpb) {
    extern __shared__ __align__(16) float lsm[];
    __shared__ uint32_t sls[LPB + 1];
    __shared__ int staged;
    float* R = lsm;                               // LCAP * dp
    float* Dt = lsm + size_t(LCAP) * dp;          // LCAP * LMAX (LMAX: 16 or 32)
    uint32_t* hI = reinterpret_cast<uint32_t*>(Dt + size_t(LCAP) * LMAX);  // k x HS
    float* hD = reinterpret_cast<float*>(hI + size_t(k) * HS);             // k x HS
    uint8_t* hF = reinterpret_cast<uint8_t*>(hD + size_t(k) * HS);         // k x HS
    __shared__ uint32_t sid[LCAP];
    __shared__ uint8_t chg[LCAP];  // the staged heap row changed
    __shared__ uint16_t sl0[LCAP], sl1[LCAP];     // leaf bounds of each staged position
    const uint32_t L0 = blockIdx.x * uint32_t(lpb);
    const uint32_t L1 = min(nleaves, L0 + uint32_t(lpb));
    const int tid = threadIdx.x;
    if (tid <= int(L1 - L0)) {
        const uint32_t li = L0 + tid;
        sls[tid] = li < nleaves ? leaf_start[li] : n;
    }
    __syncthreads();
    const uint32_t P0 = sls[0], P1 = sls[L1 - L0];
    const uint32_t span = P1 - P0;
    if (tid == 0) {
        bool ok = span <= uint32_t(LCAP);
        for (uint32_t l = 0; l < L1 - L0; ++l) ok &= sls[l + 1] - sls[l] <= uint32_t(LMAX);
        staged = ok;
    }
    __syncthreads();
    if (!staged) {
        for (uint32_t pos = P0 + tid; pos < P1; pos += LCAP) {
            uint32_t l = 0;
            while (sls[l + 1] <= pos) ++l;
            const uint32_t ls = sls[l], le = sls[l + 1];
            const uint32_t p = ids[pos];
            const float* xp = X + size_t(p) * dp;
            for (uint32_t qp = ls; qp < le; ++qp) {
                if (qp == pos) continue;
                const uint32_t q = ids[qp];
                heap_push(hidx + size_t(p) * k, hdist + size_t(p) * k, hflag + size_t(p) * k, k,
                          q, sq_dist_exact_t<D>(xp, X + size_t(q) * dp, d), 1);
            }
        }
        return;
    }
    const bool own = uint32_t(tid) < span;
    uint32_t p = 0;
    if (own) {
        p = ids[P0 + tid];
        sid[tid] = p;
        uint32_t l = 0;
        while (sls[l + 1] <= P0 + tid) ++l;
        sl0[tid] = uint16_t(sls[l] - P0);
        sl1[tid] = uint16_t(sls[l + 1] - P0);
    }
    __syncthreads();
    // rows and heap rows, all loads in flight together
    const int q4 = dp / 4;
    for (uint32_t t = tid; t < span * q4; t += LCAP) {
        const uint32_t r = t / q4, j = t - r * q4;
        reinterpret_cast<float4*>(R)[t] = reinterpret_cast<const float4*>(X + size_t(sid[r]) * dp)[j];
    }
    for (uint32_t t = tid; t < span * uint32_t(k); t += LCAP) {
        const uint32_t r = t / uint32_t(k), sl = t - r * uint32_t(k);
        const size_t g = size_t(sid[r]) * k + sl;
        hI[sl * HS + r] = hidx[g];
        hD[sl * HS + r] = hdist[g];
        hF[sl * HS + r] = hflag[g];
    }
    __syncthreads();
    if (own) {  // each pair once: this position with its later mates
        const uint32_t l0 = sl0[tid], l1 = sl1[tid];
        for (uint32_t j = tid + 1; j < l1; ++j) {
            const float dd = sq_dist_exact_t<D>(R + size_t(tid) * dp, R + size_t(j) * dp, d);
            Dt[size_t(tid) * LMAX + (j - l0)] = dd;
            Dt[size_t(j) * LMAX + (tid - l0)] = dd;
        }
    }
    __syncthreads();
    if (own) {
        const uint32_t l0 = sl0[tid], l1 = sl1[tid];
        uint32_t* ri = hI + tid;
        float* rd = hD + tid;
        uint8_t* rf = hF + tid;
        bool changed = false;
        for (uint32_t j = l0; j < l1; ++j) {
            if (j == uint32_t(tid)) continue;
            const float dd = Dt[size_t(tid) * LMAX + (j - l0)];
            if (dd >= rd[0]) continue;  // heap_push would reject it unchanged
            changed |= heap_push_strided(ri, rd, rf, k, HS, sid[j], dd, 1);
        }
        chg[tid] = changed ? 1 : 0;
    }
    __syncthreads();
    for (uint32_t t = tid; t < span * uint32_t(k); t += LCAP) {
        const uint32_t r = t / uint32_t(k), sl = t - r * uint32_t(k);
        if (!chg[r]) continue;
        const size_t g = size_t(sid[r]) * k + sl;
        hidx[g] = hI[sl * HS + r];
        hdist[g] = hD[sl * HS + r];
        hflag[g] = hF[sl * HS + r];
    }
}

__global__ void k_random_fill(const float* __restrict__ X, int d, int dp, uint32_t n, int k,
                              uint64_t seed, uint32_t* hidx, float* hdist, uint8_t* hflag) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t* ri = hidx + size_t(i) * k;
    float* rd = hdist + size_t(i) * k;
    uint8_t* rf = hflag + size_t(i) * k;
    for (uint64_t attempt = 0; attempt < 64; ++attempt) {
        bool empty = false;
        for (int s = 0; s < k; ++s) empty |= ri[s] == PQ_EMPTY;
        if (!empty) break;
        uint64_t j = hash_index(seed, uint64_t(i), attempt, n);
        if (j == i) j = (j + 1) % n;
        float dd = sq_dist_exact(X + size_t(i) * dp, X + size_t(j) * dp, d);
        heap_push(ri, rd, rf, k, uint32_t(j), dd, 1);
    }
}

}  // namespace

void launch_hyperplanes(const ForestArgs& a, PNode* nodes, uint32_t nn, float* normals,
                        cudaStream_t st) {
    k_hyper<<<nn, 64, 0, st>>>(a, nodes, normals); count_launch();
}
void launch_sides(const ForestArgs& a, const PNode* nodes, const uint32_t* chunk_node,
                  uint32_t nchunks, const float* normals, uint32_t* chunkL, cudaStream_t st) {
    const int rs = staged_stride(a.dp);
    size_t sm = size_t(a.dp) * 4, full = sm + size_t(FT) * rs * 4;
    const bool staged = full <= 100 * 1024;  // two CTAs per SM
    if (staged) sm = full;
    cudaFuncSetAttribute(k_sides, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_DYNAMIC);
    k_sides<<<nchunks, FT, sm, st>>>(a, nodes, chunk_node, normals, chunkL, staged ? rs : 0);
    count_launch();
}
void launch_node_scan(PNode* nodes, uint32_t nn, uint32_t* chunkL, cudaStream_t st) {
    k_node_scan<<<(nn + 3) / 4, 128, 0, st>>>(nodes, nn, chunkL); count_launch();
}
void launch_partition(const ForestArgs& a, PNode* nodes, const uint32_t* chunk_node,
                      uint32_t nchunks, const uint32_t* chunkPre, cudaStream_t st) {
    k_part_tables<<<nchunks, FT, 0, st>>>(a, nodes, chunk_node, chunkPre); count_launch();
    k_part_scatter<<<nchunks, FT, 0, st>>>(a, nodes, chunk_node, chunkPre); count_launch();
    k_part_copy<<<nchunks, FT, 0, st>>>(a, nodes, chunk_node); count_launch();
}
void launch_degenerate(const ForestArgs& a, PNode* nodes, uint32_t nn, cudaStream_t st) {
    k_degenerate<<<(nn + 63) / 64, 64, 0, st>>>(a, nodes, nn); count_launch();
}
void launch_leaf_compact(const uint8_t* leafflag, uint32_t T, uint32_t n, uint32_t* leaf_start,
                         uint32_t* scan_buf, void* scan_temp, uint64_t* counts, uint64_t* total,
                         cudaStream_t st) {
    const size_t tn = size_t(T) * n;
    const unsigned grid = unsigned((tn + 255) / 256);
    k_flags_u32<<<grid, 256, 0, st>>>(leafflag, tn, scan_buf); count_launch();
    scan_exclusive_u32(scan_buf, scan_buf, tn, scan_temp, total, st);
    k_leaf_scatter<<<grid, 256, 0, st>>>(leafflag, scan_buf, tn, n, leaf_start); count_launch();
    k_leaf_counts<<<(T + 63) / 64, 64, 0, st>>>(scan_buf, total, T, n, counts); count_launch();
}
void launch_leaf_pairs(const float* X, int d, int dp, const uint32_t* ids_t,
                       const uint32_t* leaf_start, uint32_t nleaves, uint32_t n, int k,
                       uint32_t leaf_cap, uint32_t* hidx, float* hdist, uint8_t* hflag,
                       cudaStream_t st) {
    if (nleaves == 0) return;
    // leaves never exceed leaf_size (or come from depth > 100); the mate table
    // is as wide as the leaf size allows (16, 32 or 64), and a CTA takes as
    // many leaves as fit its LCAP positions at that size
    int lmax = leaf_cap <= 16 ? 16 : leaf_cap <= 32 ? 32 : LMAXC;
    const int lpb = int(std::max<uint32_t>(1, std::min<uint32_t>(LPB, LCAP / std::max(leaf_cap, 1u))));
    size_t sm = leaf_pairs_smem(dp, lmax, k);
    if (sm > 200 * 1024 || leaf_cap > uint32_t(LMAXC)) {
        // wide rows, large k or large leaves: every tile takes the direct path
        lmax = 0;
        sm = 0;
    }
    const unsigned grid = (nleaves + lpb - 1) / lpb;
    if (d == 50) {
        if (sm > 40 * 1024)
            cudaFuncSetAttribute(k_leaf_pairs<50>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 SMEM_DYNAMIC);
        k_leaf_pairs<50><<<grid, LCAP, sm, st>>>(X, d, dp, ids_t, leaf_start, nleaves, n, k,
                                                 hidx, hdist, hflag, lmax, lpb); count_launch();
    } else {
        if (sm > 40 * 1024)
            cudaFuncSetAttribute(k_leaf_pairs<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 SMEM_DYNAMIC);
        k_leaf_pairs<0><<<grid, LCAP, sm, st>>>(X, d, dp, ids_t, leaf_start, nleaves, n, k,
                                                hidx, hdist, hflag, lmax, lpb); count_launch();
    }
}
void launch_random_fill(const float* X, int d, int dp, uint32_t n, int k, uint64_t seed,
                        uint32_t* hidx, float* hdist, uint8_t* hflag, cudaStream_t st) {
    k_random_fill<<<(n + 127) / 128, 128, 0, st>>>(X, d, dp, n, k, seed, hidx, hdist, hflag); count_launch();
}

}  // namespace pq
