"""A tile pass of the exact searches' filter that gives up (the bounded-wait test
hook: every CTA waits a thousand polls on an mbarrier that nothing arrives at,
before any copy or MMA).  The full search then answers every query: the bytes
of the undisturbed call, and the next call is as before."""

import ctypes as C

import numpy as np
import pytest

import oracle
import polariseq_b200 as pq
from polariseq_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def give_up(ctx):
    assert _lib.load().pq_ctx_set_test_wait(ctx._h, C.c_uint32(1000)) == _lib.PQ_OK


@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n,d,k", [(2500, 50, 15), (9000, 30, 40)])
def test_exact_search_after_an_aborted_tile_pass(metric, n, d, k):
    x = synth.mixture_dirichlet(n, d, 6, seed=n)
    ref = oracle.neighbors_exact(x, k, metric)
    ctx = pq.Context(0)
    per = k - 1
    for aborted in (False, True, False):
        if aborted:
            give_up(ctx)
        ip = np.zeros(n + 1, np.uint32)
        ix = np.zeros(n * per, np.uint32)
        dx = np.zeros(n * per, np.float32)
        assert ctx.neighbors_into(x, k, pq.METRICS[metric], ip, ix, dx) == n * per
        np.testing.assert_array_equal(ix, ref["indices"])
        assert dx.tobytes() == ref["data"].tobytes()
    ctx.close()


@pytest.mark.parametrize("graph", [True, False])
def test_batched_search_after_an_aborted_tile_pass(graph):
    import torch

    sizes, ks = [2500, 700, 4100], np.array([40, 9, 200], np.uint32)
    x = np.concatenate([synth.mixture_dirichlet(n, 30, 5, seed=n) for n in sizes])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    total = int((np.array(sizes) * ks).sum())
    ctx = pq.Context(0)
    xd = torch.from_numpy(x).cuda()

    def search(data):
        oi = torch.zeros(total, dtype=torch.int32, device="cuda")
        od = torch.zeros(total, dtype=torch.float32, device="cuda")
        ctx.knn_batched_device(data, off, ks, oi, od, graph=graph)
        torch.cuda.synchronize()
        return oi.cpu().numpy().tobytes(), od.cpu().numpy().tobytes()

    want = search(torch.nn.functional.pad(xd, (0, 33)))  # 63 dimensions: the full search
    assert search(xd) == want
    give_up(ctx)
    assert search(xd) == want
    assert search(xd) == want
    ctx.close()
