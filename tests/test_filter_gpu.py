"""The tensor-core filter of the exact searches (csrc/filter.cu) on the GPU.

The filter only decides which distances are evaluated, so its results are the
full search's, bit for bit (tolerance zero): the heap-ordered search against
the oracle, the batched search against itself with the same points in 63
dimensions (zero columns add exact zeros to every sum, and 63 dimensions take
the full search).  Sizes sit at the edges of the filter's tiles (128
candidates, 256 queries), of its range (16 points per neighbour, 512 points,
62 dimensions) and of the operand layouts (30 and 46 dimensions).
"""

import numpy as np
import pytest

import oracle
import polariseq_b200 as pq
from polariseq_b200 import synth

pytestmark = pytest.mark.gpu


def same_as_oracle(emb, k, metric):
    g = pq.neighbors_dense(emb, k, metric)
    ref = oracle.neighbors_exact(emb, k, metric)
    np.testing.assert_array_equal(g["indptr"], ref["indptr"])
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n,d,k", [
    (511, 20, 5), (512, 30, 31), (513, 31, 2), (640, 46, 15), (1025, 47, 15), (2049, 62, 31),
    (2560, 63, 15), (4113, 14, 256), (4112, 50, 256), (6000, 1, 4), (9001, 50, 15)])
def test_heap_search_edges(metric, n, d, k):
    same_as_oracle(synth.mixture_dirichlet(n, d, 12, seed=n + d), k, metric)


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_heap_search_ties_offsets_and_odd_rows(metric):
    rng = np.random.default_rng(2)
    x = synth.mixture_dirichlet(3000, 24, 6, seed=4)
    dup = x.copy()
    dup[rng.integers(0, 3000, 400)] = dup[rng.integers(0, 3000, 400)]  # equal distances
    same_as_oracle(dup, 15, metric)
    same_as_oracle(np.repeat(x[:300], 10, 0), 15, metric)              # nothing but ties
    same_as_oracle(x + np.float32(1000.0), 15, metric)                 # far from the origin
    same_as_oracle(x * np.float32(1e-20), 15, metric)                  # squares underflow
    zero = x.copy()
    zero[17] = 0.0                                                     # no cosine
    same_as_oracle(zero, 15, metric)
    order = np.argsort(x[:, 0], kind="stable")                         # sorted input
    same_as_oracle(np.ascontiguousarray(x[order]), 15, metric)


def wide(x):
    return np.ascontiguousarray(np.pad(x, ((0, 0), (0, 63 - x.shape[1]))))


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("d", [7, 30, 31, 50, 62])
def test_batched_equals_full_search(d, graph):
    rng = np.random.default_rng(d)
    sizes = [(513, 31), (700, 100), (1024, 60), (2305, 17), (9000, 512), (3000, 1), (130, 5)]
    xs = [synth.mixture_dirichlet(n, d, 5, seed=n) for n, _ in sizes]
    xs[3][rng.integers(0, 2305, 300)] = xs[3][5]  # 300 copies of one point: an overflowing list
    ks = [k for _, k in sizes]
    got = pq.knn_batched(xs, ks, graph=graph)
    ref = pq.knn_batched([wide(x) for x in xs], ks, graph=graph)
    for (gi, gd), (ri, rd) in zip(got, ref):
        np.testing.assert_array_equal(gi, ri)
        assert gd.tobytes() == rd.tobytes()


def test_batched_nonfinite_rows():
    x = synth.mixture_dirichlet(1500, 30, 5, seed=1)
    x[3, 2] = np.inf
    y = synth.mixture_dirichlet(1700, 30, 5, seed=2)
    for (gi, gd), (ri, rd) in zip(pq.knn_batched([x, y], [9, 9]),
                                  pq.knn_batched([wide(x), wide(y)], [9, 9])):
        np.testing.assert_array_equal(gi, ri)
        assert gd.tobytes() == rd.tobytes()
