"""The plan of the exact searches' tensor-core filter (csrc/filter_plan.cuh).

On the CPU the header itself is compiled and the plan walked: every chunk
maximum that the bound reads is written, and written once.  On the GPU the
batched search, whose bound needs all of the k + 1 maxima, runs at chunks of 64
to 512 columns and every remainder of the tiles by the chunk's, after a call
that leaves far larger maxima in the workspace; its results are the full
search's (the same points in 63 dimensions), bit for bit.
"""

import os
import subprocess

import numpy as np
import pytest

import polariseq_b200 as pq
from polariseq_b200 import synth

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "polariseq_b200", "csrc")

WALK = r"""
#include "filter_plan.cuh"
#include <cstdio>
#include <set>
#include <tuple>
#include <vector>
using namespace pq;
int main() {
    std::set<std::tuple<uint32_t, uint32_t>> seen;
    long plans = 0, bad = 0;
    for (uint32_t ksel : {2u, 16u, 32u, 47u, 101u, 513u})
        for (uint32_t n = 512; n <= 130000; ++n) {
            if (n < 16 * ksel) continue;
            const uint32_t tiles = (n + FILTER_TILE - 1) / FILTER_TILE;
            const uint32_t logc = filter_chunk_log(n, tiles, ksel);
            const uint32_t count = filter_chunk_count(tiles, logc);
            if (count > FILTER_MAX_CHUNKS || count < ksel) { std::printf("count n=%u\n", n); return 1; }
            if (!seen.insert({tiles, logc}).second) continue;
            for (uint32_t want : {1u, 2u, 3u, 7u, 16u}) {
                const uint32_t st = filter_slice_tiles(tiles, logc, want);
                std::vector<int> hits(count, 0);
                for (uint32_t t0 = 0; t0 < tiles; t0 += st) {
                    const uint32_t t1 = t0 + st < tiles ? t0 + st : tiles;
                    for (uint32_t t = t0; t < t1; ++t) {
                        if (logc < 7) {
                            for (uint32_t c = 0; c < (1u << (7 - logc)); ++c)
                                hits.at((t << (7 - logc)) + c)++;
                        } else if (filter_chunk_ends(t, t1, logc)) {
                            hits.at(filter_chunk_slot(t, logc))++;
                        }
                    }
                }
                ++plans;
                for (uint32_t c = 0; c < count; ++c)
                    if (hits[c] != 1) {
                        if (bad++ < 5)
                            std::printf("n=%u ksel=%u columns=%u slices of %u: chunk %u of %u written %d times\n",
                                        n, ksel, 1u << logc, st, c, count, hits[c]);
                    }
            }
        }
    std::printf("%ld plans, %ld bad\n", plans, bad);
    return bad != 0 || plans < 1000;
}
"""


def test_every_chunk_maximum_is_written_once(tmp_path):
    src, exe = tmp_path / "walk.cpp", tmp_path / "walk"
    src.write_text(WALK)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# (points, k): chunks of 64, 128, 256 and 512 columns; the tiles of the last pair
# of chunks are all of them, one, two, three or five
SIZES = [(4300, 15), (9001, 15), (9100, 15), (20000, 15), (19990, 31), (20100, 15), (20300, 15),
         (25143, 46), (32800, 7), (33400, 7)]


@pytest.mark.gpu
@pytest.mark.parametrize("d,sizes", [(12, SIZES), (50, SIZES), (50, SIZES[1:2]), (30, SIZES[3:4]),
                                     (30, SIZES[7:8])])
def test_batched_wide_chunks_after_larger_values(d, sizes):
    xs = [synth.mixture_dirichlet(n, d, 9, seed=n) for n, _ in sizes]
    ks = [k for _, k in sizes]
    pq.knn_batched([x * np.float32(1e4) for x in xs], ks)
    got = pq.knn_batched(xs, ks)
    again = pq.knn_batched(xs, ks)
    wide = [np.ascontiguousarray(np.pad(x, ((0, 0), (0, 63 - d)))) for x in xs]
    ref = pq.knn_batched(wide, ks)
    for g, a, r in zip(got, again, ref):
        for i in (0, 1):
            assert g[i].tobytes() == r[i].tobytes()
            assert a[i].tobytes() == g[i].tobytes()
