// Exact k nearest points by a tensor-core filter and exact FP32 distances.
//
// A brute-force search evaluates n distances per query in FP32 and keeps k of
// them.  Here almost none of those distances is evaluated: two passes of
// tcgen05 tiles over all pairs give every distance to within a bound (derived
// below, with one assumption about the accumulator), and only the points that can
// be among the k nearest get the search's own FP32 distance, so the result is the
// brute-force result, bit for bit.
//
//   mean, pack   coordinates centred on the group's mean (cosine: normalised
//                rows), split into two BF16 parts hi + lo;
//                candidate rows carry |x|^2 / 2 in three BF16 parts beside
//                them, query rows the constants -1, so that
//                  a = q.x - |x|^2 / 2 = (|q|^2 - |q - x|^2) / 2
//                comes out of hi.hi + lo.hi + hi.lo in one accumulator
//   pass 1       per query, the largest a of every chunk of candidates
//   bound        the (k + 1)-th largest chunk maximum: k + 1 distinct points
//                are at least that close, so nothing further than that plus
//                the error margin can be among the k nearest (one of the
//                k + 1 may be the query itself)
//   pass 2       the same tiles again; candidates above the bound are listed
//   select       FP32 distances of the listed points in the search's own
//                operation order, sorted by (distance, index)
//
// Bounds.  With A = |q|^2 - 2a and D the true squared distance, |A - D| is at
// most e s^2, s = |q| + sqrt(D) >= |x|.  A BF16 part is within 2^-8 of its value
// and the second part within 2^-17 of the binade's bottom, so dropping lo.lo and
// the two residuals leaves 2^-16 + 2 x 2^-17 of |q||x| in a: 2^-14 |q||x| in A.
// The norms' FP32 sums and the centring take 0.2e-5.  The accumulator adds the
// cross products first, at 2^-8 of the magnitude, then at most 4 K = 16 steps of
// hi.hi.  How tcgen05 rounds in between is not documented; ASSUMED is a
// truncation of each of a step's 17 terms at 2^-23 of a magnitude of at most 1.5
// s^2, 2.4e-5 in A.  Measured against FP64 (1 to 62 dimensions, both metrics,
// normal, clustered, one-sided, count and heavy-tailed values): the accumulator
// at most 1.7e-6, the sum of all 5.9e-5, against e < 8.8e-5.  The FP32 distance
// itself is within 2^-17 D (cosine: 2^-17 absolute).  The margin, 3 x 2^-14 s^2
// and those, takes both errors on both sides of the comparison; s from the bound
// itself is short by 1.4 % at most.
// A group with non-finite or huge rows, a list that overflows, an aborted
// tile pass, and (for the heap-ordered searches) equal distances among the
// k + 1 nearest send their queries to the full search.
//
// Measured at 60,013 x 30, k = 31 (Euclidean): pass 1 0.58 ms (tensor pipes 66 %
// active), bound 0.08, pass 2 0.70 (53 %), select 0.11; the full search takes 174.
// A sample with non-finite rows costs its pack and its full search only.
//
// Why two passes instead of one with running shortlists: k reaches 512, far
// past what an epilogue thread can keep in registers, and a bound known
// beforehand makes the second epilogue a compare and a rare append.  The tile
// passes are bound by the MMA issue (3 products per pair): K = 96 for d <= 30,
// 144 for d <= 46, 192 above.  256 queries per CTA halve the candidate
// traffic from L2 against 128.  Candidates are laid out in a strided order so
// that neighbouring input rows (often near-duplicates) fall into different
// chunks and slices.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <memory>
#include <numeric>

#include "ctx.cuh"
#include "filter.cuh"
#include "filter_plan.cuh"
#include "ivf.cuh"
#include "tc.cuh"

namespace pq {
namespace {

constexpr uint32_t FULL = 0xFFFFFFFFu;
constexpr int FQ = 256;              // queries per job
constexpr int FC = int(FILTER_TILE); // candidates per tile
constexpr int FEPI = 512;            // epilogue threads: 2 tile parities x 256 rows
constexpr int FNT = FEPI + 64;       // + TMA warp + MMA warp
constexpr int FROWB = 128;           // bytes per operand row and plane (64 BF16)
constexpr int FMAXCS = 6;            // candidate stages at most
constexpr int MAX_SLICES = 16;       // 2 regions per slice: one per lane of a warp
constexpr uint32_t WAIT_LIMIT = 1u << 24;

struct FBlock {       // 256 queries of one group
    uint32_t sample;  // index into the groups
    uint32_t q0;      // first query
    uint64_t min_off;   // chunk maxima: [chunk][256]
    uint64_t list_off;  // listed candidates: [256][slice][tile parity][cap]
    uint64_t cnt_off;   // list lengths: [slice][tile parity][256]
    uint32_t slot;      // first query slot of the round
    uint32_t pad;
};

struct FJob {
    uint32_t block, slice, t0, t1;  // tiles [t0, t1)
    uint32_t sample, pad;
};

struct FArgs {
    const FilterSample* samples;
    const FBlock* blocks;
    const FJob* jobs;
    uint32_t njobs;
    const int* odd;     // groups that go to the full search whole: their jobs are left out
    uint32_t plane;     // rows between the hi and lo planes (two-plane operands)
    float* minima;
    const float* ath;   // per query slot: the admission bound
    uint32_t* list;
    uint32_t* cnt;
    int* err;
    uint32_t test_wait_polls;  // pq_ctx_set_test_wait
};

struct __align__(8) FBars {
    uint64_t q_full, q_empty;
    uint64_t c_full[FMAXCS], c_empty[FMAXCS];
    uint64_t t_full[2], t_empty[2];
    uint64_t done, never;
    uint32_t tmem;
    int abort;
};

__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float fmax8(const float* v) {
    return fmax3(fmax3(v[0], v[1], v[2]), fmax3(v[3], v[4], v[5]), fmaxf(v[6], v[7]));
}

__host__ __device__ constexpr int stages(int kb) { return kb == 1 ? 6 : 4; }
constexpr size_t tile_smem(int kb) {
    return 1024 + size_t(kb) * FQ * FROWB + size_t(stages(kb)) * kb * FC * FROWB;
}

// The tile kernel of both passes: a job is 256 queries against a range of
// 128-candidate tiles.  Roles as in the shortlist kernels: a TMA warp (the
// job's query planes, candidate planes in `stages` stages), an MMA warp (two
// M = 128 halves per tile, 3 x KS K = 16 steps each, into one of two TMEM
// buffers of 256 columns) and 16 epilogue warps, 8 per TMEM buffer, each 32
// rows x 128 columns.
template <int KS, int PASS>
__global__ void __launch_bounds__(FNT, 1) k_filter_tiles(const __grid_constant__ CUtensorMap tmQ,
                                                         const __grid_constant__ CUtensorMap tmC,
                                                         FArgs a) {
    constexpr int KB = KS <= 2 ? 1 : 2;  // operand planes
    constexpr int NCS = stages(KB);
    constexpr uint32_t QPLANE = FQ * FROWB, CPLANE = FC * FROWB;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* sQ = smem;
    uint8_t* sC = sQ + KB * QPLANE;
    __shared__ FBars B;
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    volatile int* abort_flag = &B.abort;

    if (w == 0) {
        tc::tmem_alloc(&B.tmem, 512);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(&B.q_full, 1);
        tc::mbar_init(&B.q_empty, 1);
        for (int s = 0; s < NCS; ++s) {
            tc::mbar_init(&B.c_full[s], 1);
            tc::mbar_init(&B.c_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(&B.t_full[s], 1);
            tc::mbar_init(&B.t_empty[s], FEPI / 64);
        }
        tc::mbar_init(&B.done, 1);
        tc::mbar_init(&B.never, 1);
        tc::fence_barrier_init();
        B.abort = 0;
        // the timeout test hook: a bounded wait that runs out before any work
        if (a.test_wait_polls && !tc::mbar_wait(&B.never, 0, a.test_wait_polls)) B.abort = 1;
    }
    if (tid == FEPI) {
        tc::prefetch_tmap(&tmQ);
        tc::prefetch_tmap(&tmC);
    }
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t taddr = B.tmem;

    if (w == FEPI / 32) {
        // ── TMA producer ──
        if (lane == 0) {
            uint32_t qi = 0, ci = 0;
            for (uint32_t j = blockIdx.x; j < a.njobs && !*abort_flag; j += gridDim.x) {
                const FJob job = a.jobs[j];
                const int odd = a.odd[job.sample];  // (read beside the block)
                const FBlock b = a.blocks[job.block];
                const uint32_t base = uint32_t(a.samples[job.sample].base);
                if (odd) continue;
                if (!tc::mbar_wait(&B.q_empty, (qi & 1) ^ 1, WAIT_LIMIT)) {
                    *abort_flag = 1;
                    break;
                }
                tc::mbar_expect_tx(&B.q_full, KB * QPLANE);
#pragma unroll
                for (int p = 0; p < KB; ++p)
                    tc::tma_load_2d(sQ + p * QPLANE, &tmQ, &B.q_full, 0,
                                    int(uint32_t(p) * a.plane + base + b.q0));
                ++qi;
                for (uint32_t t = job.t0; t < job.t1; ++t) {
                    const int s = int(ci % NCS);
                    if (!tc::mbar_wait(&B.c_empty[s], ((ci / NCS) & 1) ^ 1, WAIT_LIMIT)) {
                        *abort_flag = 1;
                        break;
                    }
                    tc::mbar_expect_tx(&B.c_full[s], KB * CPLANE);
#pragma unroll
                    for (int p = 0; p < KB; ++p)
                        tc::tma_load_2d(sC + (s * KB + p) * CPLANE, &tmC, &B.c_full[s], 0,
                                        int(uint32_t(p) * a.plane + base + t * FC));
                    ++ci;
                }
            }
            // every issued copy has landed before the CTA may exit
            for (int s = 0; s < NCS; ++s) {
                const uint32_t uses = ci / NCS + (uint32_t(s) < ci % NCS ? 1u : 0u);
                if (uses > 0 && !tc::mbar_wait(&B.c_full[s], (uses - 1) & 1, WAIT_LIMIT))
                    *abort_flag = 1;
            }
            if (qi > 0 && !tc::mbar_wait(&B.q_full, (qi - 1) & 1, WAIT_LIMIT)) *abort_flag = 1;
        }
        __syncwarp();
    } else if (w == FEPI / 32 + 1) {
        // ── MMA issuer: the whole warp walks the jobs, so that descriptors and
        // loop counters stay warp-uniform, and one elected lane issues (a lane
        // 0 branch around the loop left 160 cycles per 64-cycle product) ──
        {
            const uint32_t idesc = tc::idesc_bf16_f32(128, FC);
            // the lo part: the next columns of the same row, or the next plane
            constexpr uint64_t QLO = KB == 1 ? uint64_t(2 * KS) : uint64_t(QPLANE >> 4);
            constexpr uint64_t CLO = KB == 1 ? uint64_t(2 * KS) : uint64_t(CPLANE >> 4);
            const uint64_t dq = tc::desc_k_sw128(tc::smem_u32(sQ));
            const uint64_t dc0 = tc::desc_k_sw128(tc::smem_u32(sC));
            uint32_t qi = 0, ci = 0, ti = 0;
            for (uint32_t j = blockIdx.x; j < a.njobs; j += gridDim.x) {
                // (one decision per warp: its lanes may read the flag apart)
                if (__any_sync(FULL, *abort_flag)) break;
                if (a.odd[a.jobs[j].sample]) continue;
                const uint32_t t0 = a.jobs[j].t0, t1 = a.jobs[j].t1;
                bool ok = __all_sync(FULL, tc::mbar_wait(&B.q_full, qi & 1, WAIT_LIMIT));
                for (uint32_t t = t0; t < t1 && ok; ++t) {
                    const uint32_t s = ci % NCS, tb = ti & 1;
                    ok = tc::mbar_wait(&B.c_full[s], (ci / NCS) & 1, WAIT_LIMIT) &&
                         tc::mbar_wait(&B.t_empty[tb], ((ti >> 1) & 1) ^ 1, WAIT_LIMIT);
                    ok = __all_sync(FULL, ok);
                    if (!ok) break;
                    tc::tc_fence_after();
                    const uint64_t dc = dc0 + uint64_t(s * (KB * CPLANE >> 4));
                    const uint32_t acc0 = taddr + tb * (2 * FC);
                    if (tc::elect_one()) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t acc = acc0 + uint32_t(h * FC);
                            const uint64_t q = dq + uint64_t(h * (128 * FROWB >> 4));
                            // the small cross products first: only the last KS
                            // steps add to an accumulator of the full magnitude
#pragma unroll
                            for (int kk = 0; kk < KS; ++kk)
                                tc::umma_f16(acc, q + QLO + 2 * kk, dc + 2 * kk, idesc,
                                             kk > 0 ? 1u : 0u);
#pragma unroll
                            for (int kk = 0; kk < KS; ++kk)
                                tc::umma_f16(acc, q + 2 * kk, dc + CLO + 2 * kk, idesc, 1u);
#pragma unroll
                            for (int kk = 0; kk < KS; ++kk)
                                tc::umma_f16(acc, q + 2 * kk, dc + 2 * kk, idesc, 1u);
                        }
                        tc::umma_commit(&B.c_empty[s]);
                        tc::umma_commit(&B.t_full[tb]);
                    }
                    __syncwarp();
                    ++ci;
                    ++ti;
                }
                if (tc::elect_one()) tc::umma_commit(&B.q_empty);
                __syncwarp();
                ++qi;
                if (!ok) {
                    *abort_flag = 1;
                    break;
                }
            }
            if (tc::elect_one()) tc::umma_commit(&B.done);
            __syncwarp();
            if (!tc::mbar_wait(&B.done, 0, WAIT_LIMIT)) *abort_flag = 1;
        }
        __syncwarp();
    } else {
        // ── epilogue: TMEM lane quarter w % 4 of row half h; the warps of group
        // grp take every other tile (the TMEM buffer grp), so that one group's
        // wait, load and filter overlap the other's ──
        const int h = (w >> 2) & 1, grp = w >> 3;
        const int row = h * 128 + (w & 3) * 32 + lane;
        const uint32_t tcol =
            taddr + (uint32_t((w & 3) * 32) << 16) + uint32_t(grp * 2 * FC + h * FC);
        const float NEG = __int_as_float(0xff800000);
        uint32_t ti = 0;  // tiles of the CTA before this job
        for (uint32_t j = blockIdx.x; j < a.njobs; j += gridDim.x) {
            if (__any_sync(FULL, *abort_flag)) break;
            const FJob job = a.jobs[j];
            const int odd = a.odd[job.sample];
            const FBlock b = a.blocks[job.block];
            const FilterSample& S = a.samples[job.sample];
            const int n = int(S.n), logc = int(S.logc);
            if (odd) continue;
            const uint32_t skip = (ti ^ uint32_t(grp)) & 1u;
            const uint32_t first = job.t0 + skip;  // this group's first tile
            const uint32_t par = first & 1u;       // all of them have this parity
            float* mrow = PASS == 1 ? a.minima + b.min_off + row : nullptr;
            float run = NEG;
            const float ath = PASS == 2 ? a.ath[b.slot + row] : 0.0f;
            const uint32_t cap = S.cap;
            uint32_t* lrow = PASS == 2 ? a.list + b.list_off +
                                             (size_t(row) * S.slices * 2 + job.slice * 2 + par) * cap
                                       : nullptr;
            uint32_t cnt = 0;
            bool ok = true;
            for (uint32_t t = first; t < job.t1; t += 2) {
                const uint32_t i = ti + (t - job.t0);
                ok = tc::mbar_wait(&B.t_full[grp], (i >> 1) & 1, WAIT_LIMIT);
                ok = __all_sync(FULL, ok);
                if (!ok) break;
                tc::tc_fence_after();
                const int lim = n - int(t * FC);  // columns that belong to the group of points
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    uint32_t r[2][32];
                    tc::tmem_ld32(tcol + uint32_t(hf * 64), r[0]);
                    tc::tmem_ld32(tcol + uint32_t(hf * 64 + 32), r[1]);
                    tc::tmem_ld_wait();
                    if (hf == 1) {  // everything is read: the buffer may be refilled
                        tc::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&B.t_empty[grp]);
                    }
                    float m64 = NEG;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int col = hf * 64 + q * 32;
                        float v[32];
#pragma unroll
                        for (int u = 0; u < 32; ++u) v[u] = __uint_as_float(r[q][u]);
                        if (lim < col + 32) {
#pragma unroll
                            for (int u = 0; u < 32; ++u)
                                if (col + u >= lim) v[u] = NEG;
                        }
                        float m8[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) m8[u] = fmax8(v + 8 * u);
                        const float m = fmaxf(fmax3(m8[0], m8[1], m8[2]), m8[3]);
                        if constexpr (PASS == 1) {
                            if (logc >= 6) {
                                m64 = fmaxf(m64, m);
                            } else if (logc == 5) {
                                mrow[size_t(t * 4 + hf * 2 + q) * FQ] = m;
                            } else if (logc == 4) {
                                mrow[size_t(t * 8 + hf * 4 + q * 2) * FQ] = fmaxf(m8[0], m8[1]);
                                mrow[size_t(t * 8 + hf * 4 + q * 2 + 1) * FQ] = fmaxf(m8[2], m8[3]);
                            } else {
#pragma unroll
                                for (int u = 0; u < 4; ++u)
                                    mrow[size_t(t * 16 + hf * 8 + q * 4 + u) * FQ] = m8[u];
                            }
                        } else {
                            if (!__any_sync(FULL, m > ath)) continue;
                            uint32_t lm = 0;
#pragma unroll
                            for (int u = 0; u < 32; ++u)
                                if (v[u] > ath) lm |= 1u << u;
                            while (lm) {
                                const int u = __ffs(lm) - 1;
                                lm &= lm - 1;
                                if (cnt < cap) lrow[cnt] = t * FC + uint32_t(col + u);
                                ++cnt;
                            }
                            __syncwarp();
                        }
                    }
                    if constexpr (PASS == 1) {
                        if (logc == 6) mrow[size_t(t * 2 + hf) * FQ] = m64;
                        else run = fmaxf(run, m64);
                    }
                }
                if constexpr (PASS == 1) {
                    if (logc >= 7 && filter_chunk_ends(t, job.t1, uint32_t(logc))) {
                        mrow[size_t(filter_chunk_slot(t, uint32_t(logc))) * FQ] = run;
                        run = NEG;
                    }
                }
            }
            if (!ok) {
                *abort_flag = 1;
                break;
            }
            ti += job.t1 - job.t0;
            if constexpr (PASS == 2)
                a.cnt[b.cnt_off + (size_t(job.slice) * 2 + par) * FQ + row] = cnt;
        }
    }
    __syncthreads();
    if (*abort_flag && tid == 0) atomicExch(a.err, 1);
    tc::tc_fence_after();
    if (w == 0) tc::tmem_dealloc(taddr, 512);
}

// The centre of each group: the mean of about 512 evenly spaced rows
// (any vector would do; a central one keeps the operands small).
__global__ void __launch_bounds__(1024) k_filter_mean(const float* __restrict__ X, int d,
                                                     const FilterSample* __restrict__ samples,
                                                     const float* __restrict__ norms,
                                                     float* __restrict__ mean) {
    __shared__ float part[32][64];
    const FilterSample S = samples[blockIdx.x];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t step = max(1u, S.n / 512u), cnt = (S.n + step - 1) / step;
    float s0 = 0.f, s1 = 0.f;
    for (uint32_t i = w; i < cnt; i += 32) {
        const uint64_t r = S.base + uint64_t(i) * step;
        const float sc = norms ? rsqrtf(norms[r]) : 1.0f;
        const float* x = X + r * uint64_t(d);
        if (lane < d) s0 += x[lane] * sc;
        if (lane + 32 < d) s1 += x[lane + 32] * sc;
    }
    part[w][lane] = s0;
    part[w][lane + 32] = s1;
    __syncthreads();
    if (threadIdx.x < 64) {
        float s = 0.f;
        for (int i = 0; i < 32; ++i) s += part[i][threadIdx.x];
        mean[size_t(blockIdx.x) * 64 + threadIdx.x] = s / float(cnt);
    }
}

// Operand rows, one warp per point: see the file comment for the columns.  A
// point's own FP32 row is copied to a 16-byte aligned row for the select
// kernel and (Xt) to a column-major copy for single queries.  Rows the bounds do not cover (non-finite or huge coordinates; for
// the cosine metric also vanishing norms) mark their group.
__global__ void __launch_bounds__(256) k_filter_pack(
    const float* __restrict__ X, int d, int dp, int db, int two_planes, uint64_t rows,
    const FilterSample* __restrict__ samples, uint32_t ns, const float* __restrict__ norms,
    const float* __restrict__ mean, __nv_bfloat16* __restrict__ Q, __nv_bfloat16* __restrict__ C,
    float* __restrict__ qn, float* __restrict__ Xp, float* __restrict__ Xt,
    int* __restrict__ odd) {
    const uint64_t t = uint64_t(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = ns;  // the last group with base <= t
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (samples[mid].base <= t) lo = mid; else hi = mid;
    }
    const FilterSample& S = samples[lo];
    if (t < S.base || t >= S.base + S.n) return;  // a group the filter does not take
    const uint64_t pos =
        S.base + (uint64_t(uint32_t(t - S.base)) * S.inv) % S.n;  // candidate position
    const float sc = norms ? norms[t] : 1.0f;
    const float rs = norms ? 1.0f / __fsqrt_rn(sc) : 1.0f;
    const uint64_t plane = rows * 64;
    float x[2], nn = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int c = lane + 32 * u;
        const float raw = c < d ? X[t * uint64_t(d) + c] : 0.0f;
        if (c < dp) Xp[t * uint64_t(dp) + c] = raw;
        if (Xt && c < d) Xt[uint64_t(c) * rows + t] = raw;
        x[u] = c < d ? raw * rs - mean[size_t(lo) * 64 + c] : 0.0f;
        nn += x[u] * x[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(FULL, nn, o);
    if (lane == 0) {
        qn[t] = nn;
        if (!(nn < 0x1p100f) || (norms && !(sc > 0x1p-100f && sc < 0x1p100f)))
            atomicExch(&odd[lo], 1);
    }
    const float h = 0.5f * nn;
    const __nv_bfloat16 h1 = __float2bfloat16_rn(h);
    const float r1 = h - __bfloat162float(h1);
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 h3 = __float2bfloat16_rn(r1 - __bfloat162float(h2));
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.f), one = __float2bfloat16_rn(-1.f);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int c = lane + 32 * u;
        if (c >= db) continue;
        const __nv_bfloat16 xh = __float2bfloat16_rn(x[u]);
        const __nv_bfloat16 xl = __float2bfloat16_rn(x[u] - __bfloat162float(xh));
        const bool p0 = c == d, p1 = c == d + 1;
        const uint64_t lo_at = two_planes ? plane + c : uint64_t(db + c);
        Q[t * 64 + c] = p0 || p1 ? one : xh;
        Q[t * 64 + lo_at] = xl;
        C[pos * 64 + c] = p0 ? h1 : p1 ? h2 : xh;
        C[pos * 64 + lo_at] = p0 ? h3 : p1 ? zero : xl;
    }
}

// Order-preserving map of a float's bits.
__device__ __forceinline__ uint32_t ford(float f) {
    const uint32_t u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float funord(uint32_t k) {
    return __uint_as_float(k & 0x80000000u ? k & 0x7FFFFFFFu : ~k);
}

// Admission bound of every query of the round: the ksel-th largest chunk
// maximum, less the margin.  One warp per query, VPL maxima per lane in
// registers, the threshold found bit by bit (the largest key, but for its
// last 8 bits, that ksel maxima reach).
template <int VPL>
__global__ void __launch_bounds__(256) k_filter_bound(const FilterSample* __restrict__ samples,
                                                      const FBlock* __restrict__ blocks,
                                                      const float* __restrict__ minima,
                                                      const float* __restrict__ qn, float abs_m,
                                                      const int* __restrict__ odd,
                                                      float* __restrict__ ath) {
    const FBlock b = blocks[blockIdx.x >> 5];
    if (odd[b.sample]) return;
    const FilterSample& S = samples[b.sample];
    const int lane = threadIdx.x & 31;
    const uint32_t row = (blockIdx.x & 31) * 8 + (threadIdx.x >> 5), q = b.q0 + row;
    if (q >= S.n) {
        if (lane == 0) ath[b.slot + row] = __int_as_float(0x7f800000);
        return;
    }
    const float* m = minima + b.min_off + row;
    uint32_t key[VPL];
#pragma unroll
    for (int t = 0; t < VPL; ++t) {
        const uint32_t c = uint32_t(t) * 32 + lane;
        key[t] = c < S.chunks ? ford(m[size_t(c) * FQ]) : 0u;
    }
    // bits above the first that differs between the extremes are common; 2^8
    // ulps are an eighth of the margin at most
    uint32_t kmax = 0, kmin = ~0u;
#pragma unroll
    for (int t = 0; t < VPL; ++t) {
        kmax = max(kmax, key[t]);
        if (uint32_t(t) * 32 + lane < S.chunks) kmin = min(kmin, key[t]);
    }
    kmax = __reduce_max_sync(FULL, kmax);
    kmin = __reduce_min_sync(FULL, kmin);
    const int top = 31 - __clz(int(kmax ^ kmin) | 0x100);
    uint32_t thr = kmin & ~((2u << top) - 1u);
    for (int bit = top; bit >= 8; --bit) {
        const uint32_t cand = thr | (1u << bit);
        uint32_t c = 0;
#pragma unroll
        for (int t = 0; t < VPL; ++t) c += key[t] >= cand ? 1u : 0u;
        c = __reduce_add_sync(FULL, c);
        if (c >= S.ksel) thr = cand;
        if (c == S.ksel) break;
    }
    if (lane == 0) {
        const float ta = funord(thr);
        const float n2 = qn[S.base + q];
        const float T = fmaxf(n2 - 2.0f * ta, 0.0f);
        const float s = sqrtf(n2) + sqrtf(T);
        const float margin = FILTER_MARGIN * s * s + 0x1p-15f * T + abs_m;
        // (a bound that is no number: everything is admitted and the list overflows)
        const float v = ta - 0.5f * margin;
        ath[b.slot + row] = v == v ? v : __int_as_float(0xff800000);
    }
}

// Ascending sort of 32 * KPL keys across the warp, key e at lane e / KPL,
// place e % KPL (bitonic network; exchanges within a lane need no shuffle).
// Up to 4 keys per lane the network is unrolled; above, its steps are loops (and
// the distances one copy of their code), which fits the instruction cache: 3 x
// 20,000 points, k = 250: 3.38 -> 2.12 ms a call, 3 x 9,000, k = 512: 1.77 ->
// 1.48, and the file compiles in 40 s instead of 320.  With loops at 2 and 4 keys
// too, 24 x 3,000 at k = 17 took 0.36 -> 0.38 ms.
template <int KPL>
__device__ __forceinline__ void sort_across(uint64_t (&v)[KPL], int lane, int ls, bool up) {
    const bool take_min = up == ((lane & ls) == 0);
#pragma unroll
    for (int t = 0; t < KPL; ++t) {
        const uint64_t o = __shfl_xor_sync(FULL, v[t], ls);
        v[t] = take_min == (o < v[t]) ? o : v[t];
    }
}
template <int KPL>
__device__ __forceinline__ void sort_within(uint64_t (&v)[KPL], int lane, int size) {
#pragma unroll
    for (int stride = KPL / 2; stride > 0; stride >>= 1) {
        if (stride >= size) continue;
#pragma unroll
        for (int t = 0; t < KPL; ++t) {
            const int u = t ^ stride;
            if (u > t) {
                const bool up = ((lane * KPL + t) & size) == 0;
                const uint64_t x = v[t], y = v[u];
                const bool sw = (x > y) == up;
                v[t] = sw ? y : x;
                v[u] = sw ? x : y;
            }
        }
    }
}
template <int KPL>
__device__ __forceinline__ void warp_sort(uint64_t (&v)[KPL], int lane) {
    if constexpr (KPL <= 4) {
#pragma unroll
        for (int size = 2; size <= 32 * KPL; size <<= 1) {
#pragma unroll
            for (int ls = size / (2 * KPL); ls > 0; ls >>= 1)
                sort_across<KPL>(v, lane, ls, ((lane * KPL) & size) == 0);
            sort_within<KPL>(v, lane, size);
        }
    } else {
#pragma unroll 1
        for (int size = 2; size <= 32 * KPL; size <<= 1) {
#pragma unroll 1
            for (int ls = size / (2 * KPL); ls > 0; ls >>= 1)
                sort_across<KPL>(v, lane, ls, ((lane * KPL) & size) == 0);
            sort_within<KPL>(v, lane, size);
        }
    }
}

struct SelArgs {
    const FilterSample* samples;
    const FBlock* blocks;
    const uint32_t* list;
    const uint32_t* cnt;
    const float* Xp;      // padded rows
    const float* norms;   // FILTER_COSINE
    int d, dp;
    int sst;              // floats between staged rows: an odd number of 16-byte units
    const int* odd;
    const int* err;
    uint32_t* out_idx;
    float* out_dist;
    // FilterCall's, for the queries that go to the full search
    const uint32_t* ids;
    const uint64_t* redo_off;
    uint32_t redo_block;
    uint32_t* redo_flag;
    uint2* redo_queries;
    uint32_t* redo_queries_n;
    uint32_t redo_short;
    uint32_t* redo_rows;
    uint32_t* redo_rows_n;
    uint32_t block0;            // first block of the launch
    // lists too long for the first launch's places: (block, row) pairs for a
    // second launch with four times the places
    uint32_t* longer;
    uint32_t* longer_n;
};

// One warp per query: the listed points' FP32 distances in the search's own
// operation order, sorted by (distance, index).  The rows of 32 candidates at a
// time come through shared memory, whole rows per load: one lane per row would
// touch 32 lines with every load (that form was bound by those wavefronts, 84
// % of the load pipe).
template <int KPL, int MODE, int D>
__device__ __forceinline__ void select_query(const SelArgs& a, uint32_t block, uint32_t row,
                                             bool second, float (*sq)[64], float* ssel) {
    const FBlock b = a.blocks[block];
    const FilterSample& S = a.samples[b.sample];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t q = b.q0 + row;
    if (q >= S.n) return;
    const uint32_t R = S.slices * 2;  // regions, at most 32
    uint32_t c = uint32_t(lane) < R ? a.cnt[b.cnt_off + size_t(lane) * FQ + row] : 0u;
    bool bad = c > S.cap || *a.err != 0 || a.odd[b.sample] != 0;
    bad = __any_sync(FULL, bad);
    uint32_t incl = bad ? 0u : c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    if (!bad && !second && total > uint32_t(32 * KPL)) {
        if (lane == 0) a.longer[atomicAdd(a.longer_n, 1u)] = block << 8 | row;
        return;
    }
    bad |= total > uint32_t(32 * KPL) || total < S.ksel;
    if (!bad) {
        const float* qr = a.Xp + (S.base + q) * uint64_t(a.dp);
        for (int t = lane; t < a.dp; t += 32) sq[w][t] = qr[t];
        __syncwarp();
        const float qnorm = MODE == FILTER_COSINE ? a.norms[S.base + q] : 0.0f;
        const uint32_t* lrow = a.list + b.list_off + size_t(row) * R * S.cap;
        const float* xb = a.Xp + S.base * uint64_t(a.dp);
        float* srow = ssel + w * 32 * a.sst;
        const int q4 = a.dp / 4;
        uint64_t v[KPL];
        // the key of element 32 t + lane (none past the list)
        auto key_of = [&](int t) -> uint64_t {
            uint64_t key = ~0ull;
            const uint32_t e = uint32_t(t) * 32 + lane;
            // the region of element e: the first whose inclusive count exceeds e
            uint32_t r = 0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const uint32_t y = __shfl_sync(FULL, incl, int(r) + o - 1);
                if (e >= y) r += uint32_t(o);
            }
            const uint32_t before = __shfl_sync(FULL, incl - c, int(r & 31u));
            uint32_t j = 0;
            if (e < total) {
                const uint32_t p = lrow[size_t(r) * S.cap + (e - before)];
                // p * stride mod n: the quotient by the reciprocal is exact or one short
                const uint64_t x = uint64_t(p) * S.stride;
                const uint64_t m = x - __umul64hi(x, S.rcp) * S.n;
                j = uint32_t(m >= S.n ? m - S.n : m);
            }
            // the 32 rows, 8 or 16 lanes per row, 16 bytes each
            __syncwarp();
            if (q4 <= 8) {
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int rr = u * 4 + (lane >> 3), cc = lane & 7;
                    const uint32_t jr = __shfl_sync(FULL, j, rr);
                    if (cc < q4)
                        *reinterpret_cast<float4*>(srow + rr * a.sst + cc * 4) =
                            *reinterpret_cast<const float4*>(xb + size_t(jr) * a.dp + cc * 4);
                }
            } else {
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const int rr = u * 2 + (lane >> 4), cc = lane & 15;
                    const uint32_t jr = __shfl_sync(FULL, j, rr);
                    if (cc < q4)
                        *reinterpret_cast<float4*>(srow + rr * a.sst + cc * 4) =
                            *reinterpret_cast<const float4*>(xb + size_t(jr) * a.dp + cc * 4);
                }
            }
            __syncwarp();
            if (e < total) {
                const float* cr = srow + lane * a.sst;
                float dd;
                if constexpr (MODE == FILTER_BATCHED) {
                    dd = 0.0f;
                    for (int u = 0; u < a.dp; u += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(&sq[w][u]);
                        const float4 y = *reinterpret_cast<const float4*>(cr + u);
                        float df = x.x - y.x;
                        dd = fmaf(df, df, dd);
                        df = x.y - y.y;
                        dd = fmaf(df, df, dd);
                        df = x.z - y.z;
                        dd = fmaf(df, df, dd);
                        df = x.w - y.w;
                        dd = fmaf(df, df, dd);
                    }
                } else if constexpr (MODE == FILTER_EUCLIDEAN) {
                    dd = sq_dist_exact_t<D>(sq[w], cr, a.d);
                } else {
                    const float dt = dot_exact_t<D>(sq[w], cr, a.d);
                    const float den =
                        __fmul_rn(__fsqrt_rn(qnorm), __fsqrt_rn(a.norms[S.base + j]));
                    dd = den > 0.0f ? __fsub_rn(1.0f, __fdiv_rn(dt, den)) : 1.0f;
                }
                if (MODE != FILTER_BATCHED || j != q) key = (uint64_t(ford(dd)) << 32) | j;
            }
            return key;
        };
        if constexpr (KPL <= 4) {
#pragma unroll
            for (int t = 0; t < KPL; ++t)
                v[t] = uint32_t(t) * 32 < total ? key_of(t) : ~0ull;  // (warp-uniform)
        } else {  // one copy of the distance's code
#pragma unroll
            for (int t = 0; t < KPL; ++t) v[t] = ~0ull;
#pragma unroll 1
            for (int t = 0; uint32_t(t) * 32 < total; ++t) {
                const uint64_t key = key_of(t);
#pragma unroll
                for (int u = 0; u < KPL; ++u) v[u] = u == t ? key : v[u];
            }
        }
        warp_sort<KPL>(v, lane);
        if constexpr (MODE != FILTER_BATCHED) {
            // equal distances among the k + 1 nearest: their order is the
            // heap's, which only the full search knows
            const uint64_t next0 = __shfl_down_sync(FULL, v[0], 1);
            bool tie = false;
#pragma unroll
            for (int t = 0; t < KPL; ++t) {
                const uint64_t nx = t + 1 < KPL ? v[t + 1 < KPL ? t + 1 : 0] : next0;
                const uint32_t p = uint32_t(lane * KPL + t);
                if (p < S.k) tie |= uint32_t(v[t] >> 32) == uint32_t(nx >> 32);
            }
            bad = __any_sync(FULL, tie);
        }
        if (!bad) {
            const int skip = MODE == FILTER_BATCHED ? 0 : 1;  // else the closest is dropped
            const int k = int(S.k);
            const uint64_t o = S.out + uint64_t(q) * uint64_t(k - skip);
#pragma unroll
            for (int t = 0; t < KPL; ++t) {
                const int p = lane * KPL + t;
                if (p >= skip && p < k) {
                    const float dd = funord(uint32_t(v[t] >> 32));
                    a.out_idx[o + (p - skip)] = uint32_t(v[t]);
                    a.out_dist[o + (p - skip)] = MODE == FILTER_COSINE ? dd : __fsqrt_rn(dd);
                }
            }
        }
    }
    if (bad && lane == 0) {
        if constexpr (MODE == FILTER_BATCHED) {
            a.redo_flag[a.redo_off[b.sample] + q / a.redo_block] = 1u;
            // (once there are too many, their number no longer matters)
            if (*static_cast<volatile uint32_t*>(a.redo_queries_n) < a.redo_short) {
                const uint32_t i = atomicAdd(a.redo_queries_n, 1u);
                if (i < a.redo_short) a.redo_queries[i] = make_uint2(a.ids[b.sample], q);
            }
        } else {
            a.redo_rows[atomicAdd(a.redo_rows_n, 1u)] = q;
        }
    }
}

// The first launch: 4 queries of one block per CTA; the second (long lists): a
// grid over the list the first launch made.
template <int KPL, int MODE, int D, bool SECOND>
__global__ void __launch_bounds__(128) k_filter_select(SelArgs a) {
    extern __shared__ __align__(16) float ssel[];  // per warp: 32 rows, sst floats apart
    __shared__ __align__(16) float sq[4][64];
    const uint32_t w = threadIdx.x >> 5;
    if constexpr (!SECOND) {
        select_query<KPL, MODE, D>(a, a.block0 + (blockIdx.x >> 6), (blockIdx.x & 63) * 4 + w,
                                   false, sq, ssel);
    } else {
        const uint32_t n = *a.longer_n;
        for (uint32_t i = blockIdx.x * 4 + w; i < n; i += gridDim.x * 4) {
            const uint32_t x = a.longer[i];
            select_query<KPL, MODE, D>(a, x >> 8, x & 255u, true, sq, ssel);
            __syncwarp();
        }
    }
}

template <int KPL, int MODE, bool SECOND>
void select_d(const SelArgs& a, uint32_t grid, cudaStream_t st) {
    const size_t sm = size_t(4) * 32 * a.sst * 4;  // at most 34 KB
    count_launch();
    if constexpr (MODE != FILTER_BATCHED) {
        if (a.d == 50) {
            k_filter_select<KPL, MODE, 50, SECOND><<<grid, 128, sm, st>>>(a);
            return;
        }
    }
    k_filter_select<KPL, MODE, 0, SECOND><<<grid, 128, sm, st>>>(a);
}
// (the second launch has four times the places of the first, 32 at most)
template <int MODE, bool SECOND>
cudaError_t launch_select(const SelArgs& a, int kpl, uint32_t grid, cudaStream_t st) {
    if constexpr (!SECOND) {
        if (kpl == 2) {
            select_d<2, MODE, SECOND>(a, grid, st);
            return cudaGetLastError();
        }
        if (kpl == 4) {
            select_d<4, MODE, SECOND>(a, grid, st);
            return cudaGetLastError();
        }
    }
    switch (kpl) {
        case 8: select_d<8, MODE, SECOND>(a, grid, st); break;
        case 16: select_d<16, MODE, SECOND>(a, grid, st); break;
        default: select_d<32, MODE, SECOND>(a, grid, st); break;
    }
    return cudaGetLastError();
}
// The select launches of one round: runs of blocks with the same first-launch
// places (groups come largest first, and k grows with the group), each
// followed by its long lists.
template <int MODE>
cudaError_t select_round(SelArgs a, const std::vector<uint8_t>& kpl, uint32_t b0, uint32_t b1,
                         cudaStream_t st) {
    for (uint32_t x = b0; x < b1;) {
        uint32_t y = x;
        while (y < b1 && kpl[y] == kpl[x]) ++y;
        cudaError_t e = cudaMemsetAsync(a.longer_n, 0, 4, st);
        if (e != cudaSuccess) return e;
        a.block0 = x - b0;
        if ((e = launch_select<MODE, false>(a, kpl[x], (y - x) * 64, st)) != cudaSuccess) return e;
        if ((e = launch_select<MODE, true>(a, std::min(32, 4 * kpl[x]), 148 * 4, st)) !=
            cudaSuccess)
            return e;
        x = y;
    }
    return cudaSuccess;
}

template <int PASS>
cudaError_t launch_tiles(int ks, const CUtensorMap& q, const CUtensorMap& c, const FArgs& a,
                         int grid, cudaStream_t st) {
    switch (ks) {
        case 1: k_filter_tiles<1, PASS><<<grid, FNT, tile_smem(1), st>>>(q, c, a); break;
        case 2: k_filter_tiles<2, PASS><<<grid, FNT, tile_smem(1), st>>>(q, c, a); break;
        case 3: k_filter_tiles<3, PASS><<<grid, FNT, tile_smem(2), st>>>(q, c, a); break;
        default: k_filter_tiles<4, PASS><<<grid, FNT, tile_smem(2), st>>>(q, c, a); break;
    }
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_bound(uint32_t max_chunks, const FilterSample* s, const FBlock* b,
                         uint32_t blocks, const float* minima, const float* qn, float abs_m,
                         const int* odd, float* ath, cudaStream_t st) {
    const unsigned g = blocks * 32;
    if (max_chunks <= 128)
        k_filter_bound<4><<<g, 256, 0, st>>>(s, b, minima, qn, abs_m, odd, ath);
    else if (max_chunks <= 512)
        k_filter_bound<16><<<g, 256, 0, st>>>(s, b, minima, qn, abs_m, odd, ath);
    else if (max_chunks <= 1024)
        k_filter_bound<32><<<g, 256, 0, st>>>(s, b, minima, qn, abs_m, odd, ath);
    else
        k_filter_bound<64><<<g, 256, 0, st>>>(s, b, minima, qn, abs_m, odd, ath);
    count_launch();
    return cudaGetLastError();
}

// Places per lane of the select kernel's first launch: a quarter more than k + 1.
int select_places(uint32_t ksel) {
    int kpl = 2;
    while (32 * kpl < int(ksel + ksel / 4 + 8)) kpl <<= 1;
    return kpl;
}

}  // namespace

bool filter_takes(uint64_t n, uint64_t d, uint64_t k) {
    return d >= 1 && d <= 62 && k >= 1 && k <= 512 && n >= 16 * (k + 1) && n >= 512 &&
           n < (uint64_t(1) << 30);
}

// A small group's search is a chain: each query is one warp that walks all
// points, 1.3 ns per point and dimension (and 12 dimensions' worth besides), 28 us
// in launches; the heap takes 3 us per neighbour.  The filter is ten launches, 80
// us whatever the group, and under the cosine metric, whose FP32 distances tie
// often, 3 us per neighbour for the queries that come back.  Whole calls, full
// search and filter: 512 x 20, k = 6, 59 and 78 us; 700 x 50, k = 2, 76 and 82;
// 1,000 x 20, k = 6, 84 and 82, cosine 92 and 108; 1,400 x 20, k = 6, 107 and 85,
// cosine 118 and 113.  With less than 28 points per neighbour a small group's bound
// is loose (8 columns per chunk at least) and its lists overflow: 512 x 20, k = 31,
// 129 and 145 us; 1,000 x 20, 170 and 84.
bool filter_pays(int mode, uint64_t n, uint64_t d, uint64_t k) {
    const uint64_t walk = n * (d + 12);
    if (mode == FILTER_COSINE) return walk + 330 * k >= 42000;
    return walk + 2300 * k >= 46000 && (n >= 896 || n >= 28 * (k + 1));
}
// The same for a batch, whose full search spreads a group over the chip: 90 us for
// the filter against 50 ns per point (90 ns above 32 dimensions) and 1.6 us per
// neighbour of the largest group beside 40 us, until the batch fills the chip.
// Whole calls without a graph: 4 x 512 x 20, k = 5, 75 and 96 us; 4 x 800 x 20, k =
// 15, 109 and 100; 30 x 512 x 20, k = 5, 123 and 137, k = 15, 171 and 140; 30 x 800,
// k = 5, 191 and 160.
bool filter_pays_batched(uint64_t points, uint64_t d, uint64_t k, uint64_t group_cost) {
    return group_cost >= 6200 || points + 500 * k >= (d <= 32 ? 20000 : 15000);
}

FilterPlan filter_prepare(pq_ctx* c, FilterCall call) {
    using pqh::ck;
    cudaStream_t st = c->stream;
    const int d = call.d, dp = (d + 3) / 4 * 4;
    const int nks = (d + 2 + 15) / 16, db = 16 * nks, kb = db <= 32 ? 1 : 2;
    const uint64_t rows = call.rows;
    std::vector<FilterSample>& S = call.samples;
    const uint32_t ns = uint32_t(S.size());
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device);

    // ── plan ──
    uint64_t qblocks = 0;
    for (const FilterSample& s : S) qblocks += (s.n + FQ - 1) / FQ;
    // enough jobs for about four per SM; a slice keeps at least two tiles
    const uint32_t want_slices =
        uint32_t(std::min<uint64_t>(MAX_SLICES, (4 * uint64_t(sms) + qblocks - 1) / qblocks));
    uint32_t max_chunks = 0;
    const uint64_t nflags = call.mode == FILTER_BATCHED ? call.redo_flags : 0;
    std::vector<uint32_t> slice_tiles(ns);
    for (uint32_t i = 0; i < ns; ++i) {
        FilterSample& s = S[i];
        s.ksel = s.k + 1;
        s.tiles = (s.n + FC - 1) / FC;
        s.logc = filter_chunk_log(s.n, s.tiles, s.ksel);
        s.chunks = filter_chunk_count(s.tiles, s.logc);
        slice_tiles[i] = filter_slice_tiles(s.tiles, s.logc, want_slices);
        s.slices = (s.tiles + slice_tiles[i] - 1) / slice_tiles[i];
        // a region's share of the admitted points is binomial around lambda
        const double lambda = 2.0 * s.ksel / (2.0 * s.slices);
        s.cap = uint32_t(std::ceil(lambda + 6.0 * std::sqrt(lambda) + 16.0));
        uint64_t stride = uint64_t(double(s.n) * 0.6180339887498949) | 1;
        while (std::gcd(stride, uint64_t(s.n)) != 1) ++stride;
        s.stride = uint32_t(stride % s.n);
        s.rcp = ~uint64_t(0) / s.n;
        // inverse of the stride modulo n (extended Euclid)
        int64_t a0 = int64_t(s.n), a1 = int64_t(s.stride), x0 = 0, x1 = 1;
        while (a1 != 0) {
            const int64_t qt = a0 / a1, a2 = a0 - qt * a1, x2 = x0 - qt * x1;
            a0 = a1;
            a1 = a2;
            x0 = x1;
            x1 = x2;
        }
        s.inv = uint32_t(x0 < 0 ? x0 + int64_t(s.n) : x0);
        max_chunks = std::max(max_chunks, s.chunks);
    }
    // groups largest first, then their query blocks, in rounds whose chunk
    // maxima and lists stay within 1.5 GB of workspace (at least one block each)
    std::vector<uint32_t> order(ns);
    std::iota(order.begin(), order.end(), 0u);
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return S[x].n > S[y].n; });
    struct Round {
        uint32_t b0, b1, j0, j1;
    };
    std::vector<Round> rounds;
    std::vector<FBlock> blocks;
    std::vector<uint8_t> kpl;  // select places of each block
    std::vector<FJob> jobs;
    uint64_t max_min = 1, max_list = 1, max_cnt = 1, max_slots = 1;
    {
        const uint64_t budget = uint64_t(1536) << 18;  // 4-byte elements
        Round r{0, 0, 0, 0};
        uint64_t um = 0, ul = 0, uc = 0, slots = 0;
        auto close = [&]() {
            r.b1 = uint32_t(blocks.size());
            r.j1 = uint32_t(jobs.size());
            if (r.b1 > r.b0) rounds.push_back(r);
            max_min = std::max(max_min, um);
            max_list = std::max(max_list, ul);
            max_cnt = std::max(max_cnt, uc);
            max_slots = std::max(max_slots, slots);
            r = Round{r.b1, 0, r.j1, 0};
            um = ul = uc = slots = 0;
        };
        for (uint32_t i : order) {
            const FilterSample& s = S[i];
            const uint64_t m = uint64_t(s.chunks) * FQ, cn = uint64_t(2) * s.slices * FQ,
                           l = cn * s.cap;
            for (uint32_t q = 0; q < s.n; q += FQ) {
                if (um + ul + m + l > budget) close();
                const uint32_t local = uint32_t(blocks.size()) - r.b0;
                blocks.push_back(FBlock{i, q, um, ul, uc, uint32_t(slots), 0});
                kpl.push_back(uint8_t(select_places(s.ksel)));
                for (uint32_t x = 0; x < s.slices; ++x)
                    jobs.push_back(FJob{local, x, x * slice_tiles[i],
                                        std::min(s.tiles, (x + 1) * slice_tiles[i]), i, 0});
                um += m;
                ul += l;
                uc += cn;
                slots += FQ;
            }
        }
        close();
    }

    // ── workspace and upload ──
    auto up = [&](const char* name, const auto& v) {
        using T = typename std::decay_t<decltype(v)>::value_type;
        T* p = c->get<T>(name, std::max<size_t>(v.size(), 1));
        if (!v.empty())
            ck(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st),
               "upload filter plan");
        return p;
    };
    FilterSample* ds = up("ft_samples", S);
    FBlock* dbk = up("ft_blocks", blocks);
    FJob* dj = up("ft_jobs", jobs);
    uint64_t* dro = up("ft_redo_off", call.redo_off);
    uint32_t* dids = up("ft_ids", call.ids);
    const uint64_t oprow = uint64_t(kb) * rows;
    __nv_bfloat16* Q = c->get<__nv_bfloat16>("ft_q", oprow * 64);
    __nv_bfloat16* C = c->get<__nv_bfloat16>("ft_c", oprow * 64);
    float* Xp = c->get<float>("ft_x", rows * dp);
    float* Xt = call.mode == FILTER_BATCHED ? nullptr : c->get<float>("ft_xt", rows * d);
    float* qn = c->get<float>("ft_qn", rows);
    float* mean = c->get<float>("ft_mean", size_t(ns) * 64);
    int* flags = c->get<int>("ft_flags", size_t(ns) + 1);  // odd groups, then the abort flag
    float* minima = c->get<float>("ft_min", max_min);
    uint32_t* list = c->get<uint32_t>("ft_list", max_list);
    uint32_t* cnt = c->get<uint32_t>("ft_cnt", max_cnt);
    float* ath = c->get<float>("ft_ath", max_slots);
    CUtensorMap tmQ, tmC;
    if (!make_bf16_map(&tmQ, Q, oprow, FQ) || !make_bf16_map(&tmC, C, oprow, FC))
        throw pqh::DeviceError{"tensor map (filter)"};
    const void* tiles[4][2] = {
        {(const void*)k_filter_tiles<1, 1>, (const void*)k_filter_tiles<1, 2>},
        {(const void*)k_filter_tiles<2, 1>, (const void*)k_filter_tiles<2, 2>},
        {(const void*)k_filter_tiles<3, 1>, (const void*)k_filter_tiles<3, 2>},
        {(const void*)k_filter_tiles<4, 1>, (const void*)k_filter_tiles<4, 2>}};
    for (const void* f : tiles[nks - 1])
        ck(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(tile_smem(kb))),
           "filter");

    FArgs fa{};
    fa.samples = ds;
    fa.plane = uint32_t(rows);
    fa.minima = minima;
    fa.ath = ath;
    fa.list = list;
    fa.cnt = cnt;
    fa.odd = flags;
    fa.err = flags + ns;
    fa.test_wait_polls = c->test_wait_polls;
    c->test_wait_polls = 0;  // the hook applies to one call
    SelArgs sa{};
    sa.samples = ds;
    sa.list = list;
    sa.cnt = cnt;
    sa.Xp = Xp;
    sa.norms = call.norms;
    sa.d = d;
    sa.dp = dp;
    sa.sst = (dp / 4) % 2 ? dp : dp + 4;
    sa.odd = flags;
    sa.err = flags + ns;
    sa.out_idx = call.out_idx;
    sa.out_dist = call.out_dist;
    sa.ids = dids;
    sa.redo_off = dro;
    sa.redo_block = call.redo_block;
    sa.redo_flag = call.redo_flag;
    sa.redo_queries = call.redo_queries;
    sa.redo_queries_n = call.redo_queries_n;
    sa.redo_short = call.redo_short;
    sa.redo_rows = call.redo_rows;
    sa.redo_rows_n = call.redo_rows_n;
    sa.longer = c->get<uint32_t>("ft_longer", max_slots);
    sa.longer_n = c->get<uint32_t>("ft_longer_n", 1);
    // the FP32 distance errs by a part of the distance (Euclidean) or by at
    // most 2^-17 of 1 - cos, 2^-16 of the squared distance (cosine), both ways
    const float abs_m = call.mode == FILTER_COSINE ? 0x1p-15f : 0x1p-110f;

    auto run = [=](cudaStream_t s) -> cudaError_t {
        cudaError_t e;
        if ((e = cudaMemsetAsync(flags, 0, (size_t(ns) + 1) * 4, s)) != cudaSuccess) return e;
        if (nflags && ((e = cudaMemsetAsync(call.redo_flag, 0, nflags * 4, s)) != cudaSuccess ||
                       (e = cudaMemsetAsync(call.redo_queries_n, 0, 4, s)) != cudaSuccess))
            return e;
        k_filter_mean<<<ns, 1024, 0, s>>>(call.X, d, ds, call.norms, mean);
        count_launch();
        k_filter_pack<<<unsigned((rows + 7) / 8), 256, 0, s>>>(
            call.X, d, dp, db, kb == 2 ? 1 : 0, rows, ds, ns, call.norms, mean, Q, C, qn, Xp, Xt,
            flags);
        count_launch();
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        for (const Round& r : rounds) {
            FArgs f = fa;
            f.blocks = dbk + r.b0;
            f.jobs = dj + r.j0;
            f.njobs = r.j1 - r.j0;
            const int grid = int(std::min<uint32_t>(f.njobs, uint32_t(sms)));
            const uint32_t nb = r.b1 - r.b0;
            if ((e = launch_tiles<1>(nks, tmQ, tmC, f, grid, s)) != cudaSuccess) return e;
            if ((e = launch_bound(max_chunks, ds, f.blocks, nb, minima, qn, abs_m, flags, ath,
                                  s)) !=
                cudaSuccess)
                return e;
            if ((e = launch_tiles<2>(nks, tmQ, tmC, f, grid, s)) != cudaSuccess) return e;
            SelArgs sel = sa;
            sel.blocks = f.blocks;
            e = call.mode == FILTER_BATCHED ? select_round<FILTER_BATCHED>(sel, kpl, r.b0, r.b1, s)
                : call.mode == FILTER_EUCLIDEAN
                    ? select_round<FILTER_EUCLIDEAN>(sel, kpl, r.b0, r.b1, s)
                    : select_round<FILTER_COSINE>(sel, kpl, r.b0, r.b1, s);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    };
    return FilterPlan{run, Xt};
}

}  // namespace pq
