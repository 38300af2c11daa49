"""Shared memory of the RP subtree kernel (csrc/seq_plan.cuh): the plan fits a
CTA for every row width that the argument rules let through (compiled with the
host compiler, on the CPU), and wide rows give the oracle's graph: staged rows
for every warp and for none, whole-row copies of 16 to 32 lanes and by the warp
in turn, and widths at which two vectors beside the rows pass a CTA's limit."""

import os
import subprocess

import numpy as np
import pytest

import oracle
import polariseq_b200 as pq
from polariseq_b200 import synth

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "polariseq_b200", "csrc")

FITS = r"""
#include "seq_plan.cuh"
#include <cstdio>
using namespace pq;
// the two CTA shapes: staged rows, room, and more static memory than they have
int main() {
    const struct { int cap; size_t room, fixed; } shape[2] = {{512, 180 * 1024, 18 * 1024},
                                                              {128, 36 * 1024, 10 * 1024}};
    int bad = 0;
    for (const auto& s : shape)
        for (int dp = 4; dp <= 25600; dp += 4) {  // 8 dp <= 200 KiB
            const int rows = seq_staged_rows(dp, s.cap, s.room, s.fixed);
            if (rows < 0 || rows > s.cap || rows == 1 ||
                s.fixed + seq_dynamic(dp, rows) > SMEM_PER_CTA) {
                if (bad++ < 5) std::printf("dp=%d cap=%d rows=%d\n", dp, s.cap, rows);
            }
            // the usual widths keep every row that the room holds
            if (dp <= 512 && rows != s.cap && size_t(rows + 1) * staged_stride(dp) * 4 <= s.room)
                ++bad;
        }
    std::printf("%d bad\n", bad);
    return bad != 0;
}
"""


def test_shared_memory_fits_at_every_width(tmp_path):
    src, exe = tmp_path / "fits.cpp", tmp_path / "fits"
    src.write_text(FITS)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,max_candidates", [
    (3000, 64, 0), (3000, 73, 0), (9000, 97, 0), (3000, 128, 0), (9000, 200, 0), (3001, 515, 0),
    (3000, 4140, 6), (2500, 5000, 5), (2200, 7000, 3), (2100, 12000, 2)])
def test_wide_rows_match_the_oracle(n, d, max_candidates):
    x = synth.mixture_dirichlet(n, d, 6, seed=d)
    g = pq.nndescent_dense(x, 10, max_candidates=max_candidates, max_iterations=3)
    ref = oracle.nndescent(x, 10, seed=0, max_candidates=max_candidates, max_iterations=3)
    np.testing.assert_array_equal(g["indptr"], ref["indptr"])
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()


@pytest.mark.gpu
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("d", [97, 512])
def test_wide_rows_exact_search(d, metric):
    x = synth.mixture_dirichlet(1500, d, 6, seed=d)
    g = pq.neighbors_dense(x, 12, metric)
    ref = oracle.neighbors_exact(x, 12, metric)
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()
