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
