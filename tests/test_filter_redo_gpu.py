"""Queries that the exact searches' filter leaves to the full search.

Batched: samples that it does not take, a sample whose rows it cannot bound (its
tiles are left out), one whose lists overflow, and ordinary ones, in one call:
the full search runs the first sample whole and of the others only the flagged
blocks, in order.  The results are the full search's alone (63 dimensions), bit
for bit.  Exact: all queries of an input with a zero row, past the first
thousand in segments of 8,192 candidates, against the oracle."""

import numpy as np
import pytest

import oracle
import polariseq_b200 as pq
from polariseq_b200 import synth

pytestmark = pytest.mark.gpu


def wide(x):
    return np.ascontiguousarray(np.pad(x, ((0, 0), (0, 63 - x.shape[1]))))


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("ks", [(20, 9, 31, 15, 40), (100, 9, 70, 15, 120)])
@pytest.mark.parametrize("odd", [True, False])
def test_batched_mixture_of_samples(graph, ks, odd):
    sizes = [2305, 100, 1900, 4001, 2600]
    xs = [synth.mixture_dirichlet(n, 30, 5, seed=n) for n in sizes]
    if odd:
        xs[0][7, 3] = np.inf
    xs[3][:] = np.tile(xs[3][:20], (201, 1))[:4001]  # 200 copies of every point
    xs[4][100:130] = xs[4][99]                       # a few queries only
    got = pq.knn_batched(xs, ks, graph=graph)
    ref = pq.knn_batched([wide(x) for x in xs], ks, graph=graph)
    for (gi, gd), (ri, rd) in zip(got, ref):
        np.testing.assert_array_equal(gi, ri)
        assert gd.tobytes() == rd.tobytes()


@pytest.mark.parametrize("n,k", [(8193, 4), (9000, 60)])
def test_exact_search_with_a_zero_row(n, k):
    x = synth.mixture_dirichlet(n, 12, 6, seed=n)
    x[17] = 0.0
    g = pq.neighbors_dense(x, k, "cosine")
    ref = oracle.neighbors_exact(x, k, "cosine")
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()


@pytest.mark.parametrize("n", [65536, 65537, 73729])
def test_exact_search_in_segments(n):
    """A huge row sends every query to the full search; in 63 dimensions (zero
    columns add exact zeros to every sum) that search runs alone."""
    x = synth.mixture_dirichlet(n, 8, 6, seed=n)
    x[17] = 1e30
    g = pq.neighbors_dense(x, 9, "euclidean")
    ref = pq.neighbors_dense(wide(x), 9, "euclidean")
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n,d,k", [
    (986, 20, 6), (1008, 20, 6), (1006, 20, 7),    # both sides of the rule at k = 6
    (672, 50, 2), (688, 50, 2), (693, 50, 3),      # and at k = 2
    (587, 30, 20), (588, 30, 20), (895, 12, 31), (896, 12, 31)])
def test_exact_search_on_both_sides_of_the_rule(metric, n, d, k):
    x = synth.mixture_dirichlet(n, d, 6, seed=n)
    g = pq.neighbors_dense(x, k, metric)
    ref = oracle.neighbors_exact(x, k, metric)
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()


@pytest.mark.parametrize("d", [32, 33])
@pytest.mark.parametrize("count,n,k", [(1, 512, 22), (1, 512, 23), (1, 1079, 5), (1, 1080, 5),
                                       (34, 512, 5), (24, 513, 5), (36, 514, 3), (30, 512, 15)])
def test_batches_on_both_sides_of_the_rule(d, count, n, k):
    xs = [synth.mixture_dirichlet(n, d, 5, seed=i) for i in range(count)]
    got = pq.knn_batched(xs, [k] * count)
    ref = pq.knn_batched([wide(x) for x in xs], [k] * count)
    for (gi, gd), (ri, rd) in zip(got, ref):
        np.testing.assert_array_equal(gi, ri)
        assert gd.tobytes() == rd.tobytes()
