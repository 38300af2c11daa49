// The RP forest below its parallel levels: every subtree is finished by one
// CTA in depth-first order with one Rng, as rp_tree_sequential /
// rp_tree_leaves (crates/polariseq-core/src/nndescent.rs:419-581) draw it, bit
// for bit.  (The partition's closed form is described in forest.cu.)
//
// A subtree is a chain: a node's draws follow those of everything left of it,
// so the time of the largest subtree bounds the phase, and within it
//   - nodes of more than `trows` points are split by the whole CTA (global
//     mode): margins of rows gathered by every warp into its own staging rows
//     (rows.cuh), sides kept as ballot words, the partition in two passes over
//     them, each warp on one contiguous run of positions, so that a node costs
//     six barriers whatever its size; ids move between the tree's two id
//     arrays instead of being copied back;
//   - a node of at most `trows` points has its ids and rows staged in shared
//     memory once (the reference gathers small subtrees for the same reason,
//     :474-491); its splits above 128 points take the whole CTA, the rest is
//     finished by warp 0 alone with ballots.
// Against the former kernel (a row per thread in the margins, block scans over
// 8-position runs, ids copied back after every split, 512-thread CTAs that left
// no room for others on their SM): 566 -> 470 ms at 4M x 50 (48 trees), 30.8 ->
// 17.7 ms at 171,003 x 30 with leaves of 30, 3.0 -> 1.8 ms at 20,000 x 50.
//
// Every thread draws from its own copy of the Rng.  The largest 148 subtrees
// run with 256 threads and 512 staged rows, beside 128-thread CTAs with 128
// staged rows for the others (256 x 128 registers leave room for two of those
// on the same SM).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "rows.cuh"
#include "seq_plan.cuh"

namespace pq {
namespace {

constexpr int STK = 128;      // depth-first stack entries (depth > 100 is a leaf)
constexpr int WCAP = 128;     // points warp 0 splits alone: 4 per lane
constexpr int WORDS = 512;    // side words of a global-mode node kept in shared memory
constexpr int BIG_NT = 256;   // threads per CTA of the largest subtrees
constexpr int BIG_CAP = 512;  // their staged points
constexpr uint32_t FULL = 0xFFFFFFFFu;

template <int NT, int CAP>
struct SeqShared {
    uint32_t stS[STK], stN[STK];  // nodes in global memory
    uint16_t stD[STK];            // depth; bit 15: the ids are in tmp
    uint32_t wst[STK], mst[STK];  // staged nodes, packed (warp 0's, the CTA's)
    uint32_t sid[CAP], sslot[CAP];
    uint32_t tabA[CAP / 2 + 1], tabB[CAP / 2 + 1];
    uint32_t lw[CAP / 32];        // left masks of a CTA split
    uint2 magic[CAP + 1];         // n: floor((2^32 - 1) / n), 2^32 mod n
    uint2 words[WORDS];           // global mode: left and tie mask per 32 positions
    uint32_t wcnt[NT / 32];
    uint8_t code[CAP];
    uint64_t rng;
    uint32_t sc;
    int sp, anytie;
};

// Staged nodes: position (10 bits), size (10 bits), depth (7 bits).
__device__ __forceinline__ uint32_t pack_node(uint32_t s, uint32_t n, uint32_t d) {
    return s | n << 10 | d << 20;
}

// The global nanosecond timer (comparable across SMs; trace only).
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// x mod n for a 32-bit x from m = floor((2^32 - 1) / n): m >= (2^32 - n) / n,
// so q = floor(x m / 2^32) > x / n - 2, i.e. q is floor(x / n) or one below,
// and one conditional subtraction of n finishes the remainder.
__device__ __forceinline__ uint32_t mod_magic(uint32_t x, uint32_t n, uint32_t m) {
    const uint32_t r = x - __umulhi(x, m) * n;
    return r >= n ? r - n : r;
}
// x mod n for n < 2^16: (hi * 2^32 + lo) mod n = ((hi mod n) * t32 + lo mod n)
// mod n with t32 = 2^32 mod n (every product and sum stays below 2^32).
__device__ __forceinline__ uint32_t mod_u64_magic(uint64_t x, uint32_t n, uint2 m) {
    const uint32_t hi = mod_magic(uint32_t(x >> 32), n, m.x), lo = mod_magic(uint32_t(x), n, m.x);
    return mod_magic(hi * m.y + lo, n, m.x);
}
__device__ __forceinline__ uint2 magic_of(uint32_t n) {
    const uint32_t m = 0xFFFFFFFFu / n, r1 = 0xFFFFFFFFu - m * n + 1u;
    return make_uint2(m, r1 == n ? 0u : r1);
}

// Draws of random_hyperplane (nndescent.rs:369-375) as positions: ids within
// a node are distinct, so the reference's `b == a` is a position test.
__device__ __forceinline__ void draw_pair(Rng& r, uint32_t n, uint32_t& pa, uint32_t& pb) {
    int tries = 0;
    if (n < 65536u) {
        const uint2 m = magic_of(n);
        pa = mod_u64_magic(r.next_u64(), n, m);
        pb = mod_u64_magic(r.next_u64(), n, m);
        while (pb == pa && tries < 8) {
            pb = mod_u64_magic(r.next_u64(), n, m);
            ++tries;
        }
        return;
    }
    const double rn = __drcp_rn(double(n));
    pa = mod_u64_u32_r(r.next_u64(), n, rn);
    pb = mod_u64_u32_r(r.next_u64(), n, rn);
    while (pb == pa && tries < 8) {
        pb = mod_u64_u32_r(r.next_u64(), n, rn);
        ++tries;
    }
}

// Element j of the normal xa - xb and of the offset's sum (its terms are
// products, so they are made in parallel and only added in order).
__device__ __forceinline__ void hyper_element(float a, float b, float* nv, float* pr) {
    const float t = __fsub_rn(a, b);
    *nv = t;
    *pr = __fmul_rn(__fmul_rn(t, 0.5f), __fadd_rn(a, b));
}
// -(sum of pr) with the reference's sequential f32 sum (folds from -0.0).
template <int D>
__device__ __forceinline__ float offset_of(const float* __restrict__ pr, int d_) {
    const int d = D > 0 ? D : d_;
    float s = -0.0f;
    int j = 0;
#pragma unroll(D > 0 ? 64 : 2)
    for (; j + 4 <= d; j += 4) {
        const float4 p = *reinterpret_cast<const float4*>(pr + j);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, p.x), p.y), p.z), p.w);
    }
    for (; j < d; ++j) s = __fadd_rn(s, pr[j]);
    return -s;
}
// dot_exact(nv, x) and offset_of(pr) in one pass (two independent chains).
template <int D>
__device__ __forceinline__ float dot_offset(const float* __restrict__ nv,
                                            const float* __restrict__ pr,
                                            const float* __restrict__ x, int d_, float& off) {
    const int d = D > 0 ? D : d_, full = d >> 3;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float s = -0.0f;
#pragma unroll(D > 0 ? 8 : 2)
    for (int c = 0; c < full; ++c) {
        const float4* n4 = reinterpret_cast<const float4*>(nv) + 2 * c;
        const float4* p4 = reinterpret_cast<const float4*>(pr) + 2 * c;
        const float4* x4 = reinterpret_cast<const float4*>(x) + 2 * c;
        const float4 n0 = n4[0], n1 = n4[1], p0 = p4[0], p1 = p4[1], y0 = x4[0], y1 = x4[1];
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, p0.x), p0.y), p0.z), p0.w);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, p1.x), p1.y), p1.z), p1.w);
        acc[0] = __fadd_rn(acc[0], __fmul_rn(n0.x, y0.x));
        acc[1] = __fadd_rn(acc[1], __fmul_rn(n0.y, y0.y));
        acc[2] = __fadd_rn(acc[2], __fmul_rn(n0.z, y0.z));
        acc[3] = __fadd_rn(acc[3], __fmul_rn(n0.w, y0.w));
        acc[4] = __fadd_rn(acc[4], __fmul_rn(n1.x, y1.x));
        acc[5] = __fadd_rn(acc[5], __fmul_rn(n1.y, y1.y));
        acc[6] = __fadd_rn(acc[6], __fmul_rn(n1.z, y1.z));
        acc[7] = __fadd_rn(acc[7], __fmul_rn(n1.w, y1.w));
    }
    float tail = 0.0f;
#pragma unroll(D > 0 ? 8 : 1)
    for (int j = full * 8; j < d; ++j) {
        s = __fadd_rn(s, pr[j]);
        tail = __fadd_rn(tail, __fmul_rn(nv[j], x[j]));
    }
    off = -s;
    const float r = __fadd_rn(__fadd_rn(__fadd_rn(acc[0], acc[4]), __fadd_rn(acc[1], acc[5])),
                              __fadd_rn(__fadd_rn(acc[2], acc[6]), __fadd_rn(acc[3], acc[7])));
    return __fadd_rn(r, tail);
}

// Side of a margin: 1 left, 0 right, 2 a tie that draws.
__device__ __forceinline__ uint32_t side_code(float m) {
    return fabsf(m) < 1e-8f ? 2u : (m > 0.0f ? 1u : 0u);
}

// Where the point at position p goes (forest.cu): lp left points before it, nL
// in all, c right points in [0, nL), n points.
__device__ __forceinline__ uint32_t partition_dst(bool left, uint32_t p, uint32_t lp, uint32_t nL,
                                                  uint32_t c, uint32_t n, const uint32_t* tA,
                                                  const uint32_t* tB) {
    if (left) return p < nL ? p : tA[nL - lp - 1];
    if (p < nL) {
        const uint32_t r = p - lp + 1;
        return (r == 1 ? n : tB[r - 2]) - 1;
    }
    if (p > nL) return p - 1;
    return (c == 0 ? n : tB[c - 1]) - 1;
}

// random_split (nndescent.rs:408-415) of n positions by one thread.
__device__ __forceinline__ void random_shuffle(Rng& rng, uint32_t n, uint32_t* ids,
                                               uint32_t* slots) {
    for (uint32_t i = n - 1; i >= 1; --i) {
        const uint32_t j = uint32_t(rng.below(uint64_t(i) + 1));
        const uint32_t t = ids[i];
        ids[i] = ids[j];
        ids[j] = t;
        if (slots) {
            const uint32_t u = slots[i];
            slots[i] = slots[j];
            slots[j] = u;
        }
    }
}

// Warp 0 splits a staged node of at most 32 * G points: positions [0, n) of
// sid / sslot, rows in `rows` (slot-indexed).  la1 and la2 are the next two
// Rng states, computed while the previous split works.  Returns the split.
template <int G, int D, class SS>
__device__ __forceinline__ uint32_t warp_split(const ForestArgs& a, SS& S, uint32_t* sid,
                                               uint32_t* sslot, const float* rows, int rs,
                                               float* nv, float* pr, uint32_t n, Rng& rng,
                                               uint64_t& la1, uint64_t& la2) {
    const uint32_t lane = threadIdx.x & 31, last = n - 1;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t id[G], sl[G];
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const uint32_t q = min(lane + 32u * i, last);
        id[i] = sid[q];
        sl[i] = sslot[q];
    }
    const uint2 mg = S.magic[n];
    const uint32_t pa = mod_u64_magic(la1, n, mg);
    uint32_t pb = mod_u64_magic(la2, n, mg);
    rng.s = la2;
    for (int tries = 0; pb == pa && tries < 8; ++tries) pb = mod_u64_magic(rng.next_u64(), n, mg);
    const float* xa = rows + sslot[pa] * rs;
    const float* xb = rows + sslot[pb] * rs;
    for (int e = int(lane); e < (D > 0 ? D : a.d); e += 32)
        hyper_element(xa[e], xb[e], nv + e, pr + e);
    la1 = splitmix(rng.s);
    la2 = splitmix(la1);
    __syncwarp();
    float dots[G], off;
    dots[0] = dot_offset<D>(nv, pr, rows + sl[0] * rs, a.d, off);
#pragma unroll
    for (int i = 1; i < G; ++i) dots[i] = dot_exact_t<D>(nv, rows + sl[i] * rs, a.d);
    uint32_t code[G];
    bool tie = false;
#pragma unroll
    for (int i = 0; i < G; ++i) {
        code[i] = lane + 32u * i < n ? side_code(__fadd_rn(dots[i], off)) : 0u;
        tie |= code[i] == 2;
    }
    if (__any_sync(FULL, tie)) {
        // ties draw from the Rng in position order (every lane replays the
        // same draws so that all copies of the Rng stay equal)
        if (a.trace && lane == 0) atomicAdd(&a.trace[SEQ_T_TIES], 1ull);
#pragma unroll
        for (int i = 0; i < G; ++i)
            if (lane + 32u * i < n) S.code[lane + 32u * i] = uint8_t(code[i]);
        __syncwarp();
        for (uint32_t p = 0; p < n; ++p)
            if (S.code[p] == 2) {
                const uint8_t v = (rng.next_u64() & 1ull) == 0 ? 1 : 0;
                __syncwarp();
                if (lane == 0) S.code[p] = v;
                __syncwarp();
            }
#pragma unroll
        for (int i = 0; i < G; ++i)
            if (lane + 32u * i < n) code[i] = S.code[lane + 32u * i];
        la1 = splitmix(rng.s);  // the tie draws moved the Rng on
        la2 = splitmix(la1);
    }
    unsigned mask[G];
    uint32_t nL = 0;
#pragma unroll
    for (int i = 0; i < G; ++i) {
        mask[i] = __ballot_sync(FULL, code[i] == 1);
        nL += __popc(mask[i]);
    }
    // the moved points of the two sides meet through the rank tables
    uint32_t lp[G], pre = 0, c = 0;
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const uint32_t p = lane + 32u * i;
        lp[i] = pre + __popc(mask[i] & lt);
        if (p < n) {
            if (code[i] == 1) {
                if (p >= nL) S.tabB[nL - lp[i] - 1] = p;
            } else if (p < nL) {
                S.tabA[p - lp[i]] = p;
            }
        }
        // c = right points in [0, nL) = nL - (left points in [0, nL))
        if (nL >= 32u * i && nL < 32u * i + 32u)
            c = nL - (pre + __popc(mask[i] & ((1u << (nL - 32u * i)) - 1u)));
        pre += __popc(mask[i]);
    }
    __syncwarp();  // (every lane read its ids and slots before this)
#pragma unroll
    for (int i = 0; i < G; ++i) {
        const uint32_t p = lane + 32u * i;
        if (p < n) {
            const uint32_t dst = partition_dst(code[i] == 1, p, lp[i], nL, c, n, S.tabA, S.tabB);
            sid[dst] = id[i];
            sslot[dst] = sl[i];
        }
    }
    __syncwarp();
    if (nL == 0 || nL == n) {
        if (a.trace && lane == 0) atomicAdd(&a.trace[SEQ_T_DEGENERATE], 1ull);
        if (lane == 0) random_shuffle(rng, n, sid, sslot);
        rng.s = __shfl_sync(FULL, rng.s, 0);
        __syncwarp();
        nL = n / 2;
        la1 = splitmix(rng.s);  // the random split moved the Rng on
        la2 = splitmix(la1);
    }
    return nL;
}

// Warp 0 finishes a staged subtree of at most WCAP points: local positions
// [0, n0); `leaf` points at its first position's flag.  Leaves are flagged as
// their parent is split; the left child is split next from registers, right
// children wait on the stack.
template <int D, class SS>
__device__ void warp_subtree(const ForestArgs& a, SS& S, uint32_t* sid, uint32_t* sslot,
                             const float* rows, int rs, float* nv, float* pr, uint32_t n0,
                             uint32_t d0, Rng& rng, uint8_t* leaf) {
    const int lane = threadIdx.x & 31;
    uint64_t la1 = splitmix(rng.s), la2 = splitmix(la1);
    uint32_t ls = 0, ln = n0, ld = d0;
    int sp = 0;
    uint32_t nodes = 0;
    for (;;) {
        uint32_t split;
        if (ln <= 32)
            split = warp_split<1, D>(a, S, sid + ls, sslot + ls, rows, rs, nv, pr, ln, rng, la1, la2);
        else if (ln <= 64)
            split = warp_split<2, D>(a, S, sid + ls, sslot + ls, rows, rs, nv, pr, ln, rng, la1, la2);
        else
            split = warp_split<4, D>(a, S, sid + ls, sslot + ls, rows, rs, nv, pr, ln, rng, la1, la2);
        ++nodes;
        const bool deep = ld + 1 > 100;
        const bool lleaf = split <= a.leaf_size || deep, rleaf = ln - split <= a.leaf_size || deep;
        if (lane == 0) {
            if (lleaf) leaf[ls] = 1;
            if (rleaf) leaf[ls + split] = 1;
        }
        if (!lleaf) {
            if (!rleaf) {
                if (lane == 0) S.wst[sp] = pack_node(ls + split, ln - split, ld + 1);
                ++sp;  // (at most one entry per level below d0)
            }
            ln = split;
            ++ld;
        } else if (!rleaf) {
            ls += split;
            ln -= split;
            ++ld;
        } else {
            if (sp == 0) break;
            __syncwarp();
            const uint32_t x = S.wst[--sp];
            __syncwarp();
            ls = x & 1023u;
            ln = (x >> 10) & 1023u;
            ld = x >> 20;
        }
    }
    if (a.trace && lane == 0) atomicAdd(&a.trace[SEQ_T_STAGED_NODES], (unsigned long long)nodes);
}

// One split of a staged node of n <= BIG_CAP points by the whole CTA, two
// positions per thread.  Returns the split.
template <int NT, int D, class SS>
__device__ uint32_t cta_split(const ForestArgs& a, SS& S, uint32_t* sid, uint32_t* sslot,
                              uint32_t n, Rng& rng, const float* rows, int rs, float* nv,
                              float* pr) {
    constexpr int U = BIG_CAP / NT, NG = BIG_CAP / 32;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint2 mg = S.magic[n];
    const uint32_t pa = mod_u64_magic(rng.next_u64(), n, mg);
    uint32_t pb = mod_u64_magic(rng.next_u64(), n, mg);
    for (int tries = 0; pb == pa && tries < 8; ++tries) pb = mod_u64_magic(rng.next_u64(), n, mg);
    const float* xa = rows + sslot[pa] * rs;
    const float* xb = rows + sslot[pb] * rs;
    for (int e = int(tid); e < a.d; e += NT) hyper_element(xa[e], xb[e], nv + e, pr + e);
    uint32_t id[U], sl[U], code[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t q = min(tid + uint32_t(u * NT), n - 1);
        id[u] = sid[q];
        sl[u] = sslot[q];
    }
    __syncthreads();
    float off, dots[U];
    dots[0] = dot_offset<D>(nv, pr, rows + sl[0] * rs, a.d, off);
    bool tie = false;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        code[u] = 0;
        if (u > 0 && w * 32 + uint32_t(u * NT) < n)  // warp-uniform
            dots[u] = dot_exact_t<D>(nv, rows + sl[u] * rs, a.d);
        if (tid + uint32_t(u * NT) < n) code[u] = side_code(__fadd_rn(dots[u], off));
        tie |= code[u] == 2;
        const unsigned m = __ballot_sync(FULL, code[u] == 1);
        if (lane == 0) S.lw[w + u * (NT / 32)] = m;
    }
    if (__syncthreads_or(tie)) {
        // ties draw from the Rng in position order (every thread replays the
        // same draws)
        if (a.trace && tid == 0) atomicAdd(&a.trace[SEQ_T_TIES], 1ull);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (tid + uint32_t(u * NT) < n) S.code[tid + u * NT] = uint8_t(code[u]);
        __syncthreads();
        for (uint32_t q = 0; q < n; ++q)
            if (S.code[q] == 2) {
                const uint32_t v = (rng.next_u64() & 1ull) == 0 ? 1u : 0u;
                if (tid == 0 && v) S.lw[q >> 5] |= 1u << (q & 31);
            }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < U; ++u) code[u] = (S.lw[w + u * (NT / 32)] >> lane) & 1u;
    }
    // left points before every group of 32: each warp scans the masks itself
    uint32_t v = lane < uint32_t(NG) ? __popc(S.lw[lane < uint32_t(NG) ? lane : 0]) : 0u;
#pragma unroll
    for (int o = 1; o < NG; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, v, o);
        if (lane >= uint32_t(o)) v += y;
    }
    const uint32_t nL = __shfl_sync(FULL, v, NG - 1);
    uint32_t lp[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t g = w + u * (NT / 32), p = tid + u * NT;
        const uint32_t before = __shfl_sync(FULL, v, g > 0 ? int(g) - 1 : 0);
        lp[u] = (g > 0 ? before : 0u) + __popc(S.lw[g] & ((1u << lane) - 1u));
        if (p < n) {
            if (code[u] == 1) {
                if (p >= nL) S.tabB[nL - lp[u] - 1] = p;
            } else if (p < nL) {
                S.tabA[p - lp[u]] = p;
            }
            if (p == nL) S.sc = nL - lp[u];  // right points in [0, nL)
        }
    }
    __syncthreads();  // (every thread read its ids and slots before this)
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const uint32_t p = tid + u * NT;
        if (p < n) {
            const uint32_t dst = partition_dst(code[u] == 1, p, lp[u], nL, S.sc, n, S.tabA, S.tabB);
            sid[dst] = id[u];
            sslot[dst] = sl[u];
        }
    }
    __syncthreads();
    uint32_t split = nL;
    if (nL == 0 || nL == n) {
        if (a.trace && tid == 0) atomicAdd(&a.trace[SEQ_T_DEGENERATE], 1ull);
        if (tid == 0) {
            random_shuffle(rng, n, sid, sslot);
            S.rng = rng.s;
        }
        __syncthreads();
        rng.s = S.rng;
        split = n / 2;
    }
    return split;
}

// A staged subtree of sz points, ids src[0, sz), the first at position gpos of
// the tree: ids and rows are staged once, its nodes of more than WCAP points
// split by the whole CTA, the smaller ones finished by warp 0; the ids go to
// dst in tree order.
template <int NT, int CAP, int D, class SS>
__device__ void staged_subtree(const ForestArgs& a, SS& S, const uint32_t* src, uint32_t* dst,
                               uint32_t sz, uint32_t dep, Rng& rng, float* rows, int rs, float* nv,
                               float* pr, uint8_t* leaf, bool tb0) {
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    for (uint32_t g = w * 32; g < sz; g += NT) {
        const uint32_t p = g + lane;
        const uint32_t id = src[min(p, sz - 1)];
        if (p < sz) {
            S.sid[p] = id;
            S.sslot[p] = p;
        }
        warp_stage_rows(a.X, a.dp, rs, id, min(32u, sz - g), rows + size_t(g) * rs);
    }
    cp_async_commit();
    cp_async_wait<0>();
    int sp = 0;
    uint32_t ls = 0, ln = sz, ld = dep;
    __syncthreads();
    for (;;) {
        bool pop = true;
        if (ln <= a.leaf_size || ld > 100) {
            if (tid == 0) leaf[ls] = 1;
        } else if (CAP <= WCAP || ln <= uint32_t(WCAP)) {
            if (tid < 32) {
                const long long c0 = tb0 ? clock64() : 0;
                warp_subtree<D>(a, S, S.sid + ls, S.sslot + ls, rows, rs, nv, pr, ln, ld, rng,
                                leaf + ls);
                if (tid == 0) S.rng = rng.s;
                if (tb0) a.trace[SEQ_T_R0_CYC_WARP] += clock64() - c0;
            }
            __syncthreads();
            rng.s = S.rng;  // the other warps adopt warp 0's Rng state
        } else {
            if (a.trace && tid == 0) atomicAdd(&a.trace[SEQ_T_MID_NODES], 1ull);
            const uint32_t split =
                cta_split<NT, D>(a, S, S.sid + ls, S.sslot + ls, ln, rng, rows, rs, nv, pr);
            // every thread keeps the walk itself; right children on the stack
            // (at most one per level)
            if (tid == 0) S.mst[sp] = pack_node(ls + split, ln - split, ld + 1);
            ++sp;
            ln = split;
            ++ld;
            pop = false;
        }
        if (pop) {
            if (sp == 0) break;
            __syncthreads();
            const uint32_t x = S.mst[--sp];
            __syncthreads();
            ls = x & 1023u;
            ln = (x >> 10) & 1023u;
            ld = x >> 20;
        }
    }
    __syncthreads();
    for (uint32_t p = tid; p < sz; p += NT) dst[p] = S.sid[p];
    __syncthreads();
    if (a.trace && tid == 0) atomicAdd(&a.trace[SEQ_T_STAGED_TREES], 1ull);
}

// One node split in global mode: positions [st, st + sz) of src, partitioned
// into dst.  `rows` holds `stages` groups of 32 staged rows per warp (none: a
// thread reads its own row).  Returns the split.
template <int NT, int D, class SS>
__device__ uint32_t split_node(const ForestArgs& a, SS& S, const uint32_t* src, uint32_t* dst,
                               uint8_t* side, uint32_t* tabA, uint32_t* tabB, uint32_t st,
                               uint32_t sz, Rng& rng, float* nv, float* pr, float* rows, int rs,
                               int stages, uint32_t room, bool tb0, long long& tclk) {
    constexpr uint32_t NW = NT / 32;
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int d = a.d, dp = a.dp;
    unsigned long long* tr = a.trace;
    auto phase = [&](int slot) {
        if (tb0) {
            const long long t1 = clock64();
            tr[slot] += t1 - tclk;
            tclk = t1;
        }
    };
    if (tr && tid == 0) {
        atomicAdd(&tr[SEQ_T_GLOBAL_NODES], 1ull);
        atomicAdd(&tr[SEQ_T_GLOBAL_POINTS], (unsigned long long)sz);
    }
    src += st;
    dst += st;
    const uint32_t groups = (sz + 31) / 32, gpw = (groups + NW - 1) / NW;
    const uint32_t g0 = min(w * gpw, groups), g1 = min(g0 + gpw, groups);
    // the first rows are on their way before the hyperplane is known
    auto id_at = [&](uint32_t g) { return src[min(g * 32 + lane, sz - 1)]; };
    float* mine = rows + size_t(w) * uint32_t(stages) * 32 * rs;
    uint32_t idn[2] = {0, 0};  // ids of the next two groups
    if (g0 < g1) idn[0] = id_at(g0);
    if (g0 + 1 < g1) idn[1] = id_at(g0 + 1);
    uint32_t pa, pb;
    draw_pair(rng, sz, pa, pb);
    {
        const uint32_t A = src[pa], B = src[pb];
        if (stages > 0) {
            if (g0 < g1) warp_stage_rows(a.X, dp, rs, idn[0], min(32u, sz - g0 * 32), mine);
            cp_async_commit();
            if (stages > 1) {
                if (g0 + 1 < g1)
                    warp_stage_rows(a.X, dp, rs, idn[1], min(32u, sz - (g0 + 1) * 32),
                                    mine + 32 * rs);
                cp_async_commit();
            }
        }
        for (int e = int(tid); e < d; e += NT)
            hyper_element(a.X[size_t(A) * dp + e], a.X[size_t(B) * dp + e], nv + e, pr + e);
    }
    if (tid == 0) {
        S.anytie = 0;
        S.sc = 0;
    }
    __syncthreads();
    const float off = offset_of<D>(pr, d);
    phase(SEQ_T_CYC_DRAW);
    // side words: left and tie mask of every 32 positions
    uint2* words = S.words;
    if (groups > uint32_t(WORDS))
        words = reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(side + st) + 7) & ~uintptr_t(7));
    uint32_t cnt = 0, ties = 0;
    auto sides = [&](uint32_t g, const float* x) {
        uint32_t code = 0;
        if (g * 32 + lane < sz) code = side_code(__fadd_rn(dot_exact_t<D>(nv, x, d), off));
        const unsigned l = __ballot_sync(FULL, code == 1), t = __ballot_sync(FULL, code == 2);
        if (lane == 0) words[g] = make_uint2(l, t);
        cnt += __popc(l);
        ties |= t;
    };
    if (stages >= 2) {
        // group g in one stage while the next is copied into the other
        uint32_t id2 = g0 + 2 < g1 ? id_at(g0 + 2) : 0u;
        for (uint32_t g = g0; g < g1; ++g) {
            const uint32_t id3 = g + 3 < g1 ? id_at(g + 3) : 0u;
            float* buf = mine + ((g - g0) & 1u) * 32 * rs;
            cp_async_wait<1>();
            __syncwarp();
            sides(g, buf + lane * rs);
            __syncwarp();
            if (g + 2 < g1) warp_stage_rows(a.X, dp, rs, id2, min(32u, sz - (g + 2) * 32), buf);
            cp_async_commit();
            id2 = id3;
        }
        cp_async_wait<0>();
    } else if (stages == 1) {
        uint32_t id1 = idn[1];
        for (uint32_t g = g0; g < g1; ++g) {
            const uint32_t id2 = g + 2 < g1 ? id_at(g + 2) : 0u;
            cp_async_wait<0>();
            __syncwarp();
            sides(g, mine + lane * rs);
            __syncwarp();
            if (g + 1 < g1) warp_stage_rows(a.X, dp, rs, id1, min(32u, sz - (g + 1) * 32), mine);
            cp_async_commit();
            id1 = id2;
        }
        cp_async_wait<0>();
    } else {
        for (uint32_t g = g0; g < g1; ++g) sides(g, a.X + size_t(id_at(g)) * dp);
    }
    if (lane == 0) {
        S.wcnt[w] = cnt;
        if (ties) S.anytie = 1;
    }
    __syncthreads();
    phase(SEQ_T_CYC_MARGIN);
    if (S.anytie) {
        // ties draw from the Rng in position order; every thread replays the
        // draws, thread 0 writes the sides
        if (tr && tid == 0) atomicAdd(&tr[SEQ_T_TIES], 1ull);
        for (uint32_t g = 0; g < groups; ++g) {
            uint32_t add = 0;
            for (uint32_t t = words[g].y; t; t &= t - 1)
                if ((rng.next_u64() & 1ull) == 0) add |= t & (0u - t);
            if (tid == 0 && add) words[g].x |= add;
        }
        __syncthreads();
        cnt = 0;
        for (uint32_t g = g0 + lane; g < g1; g += 32) cnt += __popc(words[g].x);
        cnt = __reduce_add_sync(FULL, cnt);
        if (lane == 0) S.wcnt[w] = cnt;
        __syncthreads();
    }
    uint32_t nL = 0, pre = 0;
#pragma unroll
    for (uint32_t i = 0; i < NW; ++i) {
        if (i == w) pre = nL;
        nL += S.wcnt[i];
    }
    // rank tables, in the staging rows where they fit (each holds at most
    // min(nL, sz - nL) positions)
    uint32_t *tA = tabA + st, *tB = tabB + st;
    if (room >= sz + 2) {
        tA = reinterpret_cast<uint32_t*>(rows);
        tB = tA + (sz / 2 + 1);
    }
    const unsigned lt = (1u << lane) - 1u;
    uint32_t run = pre;
    for (uint32_t g = g0; g < g1; ++g) {
        const uint32_t l = words[g].x, p = g * 32 + lane, lp = run + __popc(l & lt);
        if (p < sz) {
            if ((l >> lane) & 1u) {
                if (p >= nL) tB[nL - lp - 1] = p;
            } else if (p < nL) {
                tA[p - lp] = p;
            }
            if (p == nL) S.sc = nL - lp;
        }
        run += __popc(l);
    }
    __syncthreads();
    const uint32_t c = S.sc;
    run = pre;
#pragma unroll 2
    for (uint32_t g = g0; g < g1; ++g) {
        const uint32_t l = words[g].x, p = g * 32 + lane, lp = run + __popc(l & lt);
        if (p < sz) dst[partition_dst((l >> lane) & 1u, p, lp, nL, c, sz, tA, tB)] = src[p];
        run += __popc(l);
    }
    __syncthreads();
    uint32_t split = nL;
    if (nL == 0 || nL == sz) {
        if (tr && tid == 0) atomicAdd(&tr[SEQ_T_DEGENERATE], 1ull);
        if (tid == 0) {
            random_shuffle(rng, sz, dst, nullptr);
            S.rng = rng.s;
        }
        __syncthreads();
        rng.s = S.rng;
        split = sz / 2;
    }
    phase(SEQ_T_CYC_PART);
    return split;
}

template <int NT, int CAP, int D>
__global__ void __launch_bounds__(NT, NT == BIG_NT ? 2 : 5)
    k_seqtree(ForestArgs a, const SRoot* roots, int trows) {
    extern __shared__ __align__(16) float dyn[];
    __shared__ SeqShared<NT, CAP> S;
    const int rs = staged_stride(a.dp);
    float* nv = dyn;             // dp: the normal
    float* pr = dyn + a.dp;      // dp: the offset's terms
    float* rows = dyn + 2 * a.dp;  // trows * rs
    const int stages = trows / NT;  // groups of 32 staged rows per warp
    const uint32_t room = uint32_t(trows) * uint32_t(rs);
    const uint32_t tid = threadIdx.x;
    const SRoot rt = roots[blockIdx.x];
    const size_t tb = size_t(rt.tree) * a.n;
    uint32_t* ids = a.ids + tb;
    uint32_t* tmp = a.tmp + tb;
    uint8_t* leaf = a.leafflag + tb;
    Rng rng{rt.seed};  // every thread holds the same state
    unsigned long long* tr = a.trace;
    const bool tb0 = tr && rt.size == tr[SEQ_T_ROOT0] && tid == 0;
    long long t_start = clock64(), tclk = 0;
    const unsigned long long g_start = a.tl ? globaltimer_ns() : 0ull;
    for (uint32_t i = tid + 1; i <= uint32_t(CAP); i += NT) S.magic[i] = magic_of(i);
    if (tid == 0) {
        S.sp = 1;
        S.stS[0] = rt.start;
        S.stN[0] = rt.size;
        S.stD[0] = uint16_t(rt.depth);
    }
    __syncthreads();
    while (S.sp > 0) {
        const uint32_t st = S.stS[S.sp - 1], sz = S.stN[S.sp - 1], de = S.stD[S.sp - 1];
        const uint32_t dep = de & 0x7FFFu;
        const bool in_tmp = de >> 15;
        const uint32_t* src = in_tmp ? tmp : ids;
        __syncthreads();
        if (tid == 0) S.sp -= 1;
        if (sz <= a.leaf_size || dep > 100) {
            if (tid == 0) leaf[st] = 1;
            if (in_tmp)
                for (uint32_t p = tid; p < sz; p += NT) ids[st + p] = tmp[st + p];
            __syncthreads();
            continue;
        }
        if (tb0) tclk = clock64();
        if (sz <= uint32_t(trows)) {
            staged_subtree<NT, CAP, D>(a, S, src + st, ids + st, sz, dep, rng, rows, rs, nv, pr,
                                       leaf + st, tb0);
            if (tb0) tr[SEQ_T_CYC_STAGED] += clock64() - tclk;
            continue;
        }
        const uint32_t split =
            split_node<NT, D>(a, S, src, in_tmp ? ids : tmp, a.side + tb, a.tabA + tb, a.tabB + tb,
                              st, sz, rng, nv, pr, rows, rs, stages, room, tb0, tclk);
        if (tid == 0) {
            const uint32_t cd = (dep + 1) | (in_tmp ? 0u : 0x8000u);
            if (S.sp + 2 > STK) {
                atomicExch(a.err, 1);
                S.sp = 0;
            } else {
                S.stS[S.sp] = st + split;  // right, popped after the whole left subtree
                S.stN[S.sp] = sz - split;
                S.stD[S.sp] = uint16_t(cd);
                S.stS[S.sp + 1] = st;
                S.stN[S.sp + 1] = split;
                S.stD[S.sp + 1] = uint16_t(cd);
                S.sp += 2;
            }
        }
        __syncthreads();
    }
    if (tb0) tr[SEQ_T_CYC_TOTAL] = clock64() - t_start;
    if (a.tl && tid == 0) {
        unsigned long long* tl = a.tl;
        const unsigned long long g_end = globaltimer_ns();
        if (NT == BIG_NT) {
            if (blockIdx.x < unsigned(SEQ_T_BIG_N)) {
                tl[SEQ_T_BIG + 2 * blockIdx.x] = g_start;
                tl[SEQ_T_BIG + 2 * blockIdx.x + 1] = g_end;
            }
        } else {
            atomicMax(&tl[SEQ_T_SMALL_T0], ~g_start);  // the earliest start, complemented
            atomicMax(&tl[SEQ_T_SMALL_T1], g_end);
        }
    }
}

// Static shared memory of a subtree CTA (with room for the compiler's alignment).
template <int NT, int CAP>
constexpr size_t SEQ_FIXED = sizeof(SeqShared<NT, CAP>) + 64;

template <int NT, int CAP, int D>
void seqtree_launch(const ForestArgs& a, const SRoot* roots, uint32_t nr, size_t room,
                    cudaStream_t st) {
    if (nr == 0) return;
    const int trows = seq_staged_rows(a.dp, CAP, room, SEQ_FIXED<NT, CAP>);
    const size_t dyn = seq_dynamic(a.dp, trows);
    // (with the static arrays the total passes 48 KB well before dyn does)
    cudaFuncSetAttribute(k_seqtree<NT, CAP, D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(SMEM_PER_CTA - SEQ_FIXED<NT, CAP>));
    k_seqtree<NT, CAP, D><<<nr, NT, dyn, st>>>(a, roots, trows);
    count_launch();
}

}  // namespace

void launch_seqtrees(const ForestArgs& a, const SRoot* roots, uint32_t n_big, uint32_t nr,
                     cudaStream_t st, cudaStream_t st_big) {
    if (nr == 0) return;
    if (a.d == 50) {
        seqtree_launch<BIG_NT, BIG_CAP, 50>(a, roots, n_big, 180 * 1024, st_big);
        seqtree_launch<128, WCAP, 50>(a, roots + n_big, nr - n_big, 36 * 1024, st);
    } else {
        seqtree_launch<BIG_NT, BIG_CAP, 0>(a, roots, n_big, 180 * 1024, st_big);
        seqtree_launch<128, WCAP, 0>(a, roots + n_big, nr - n_big, 36 * 1024, st);
    }
}

}  // namespace pq
