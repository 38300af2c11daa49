"""The filter's workspace is optional: it makes room for a call that needs the
memory, and a set-up that does not find room gives back what it got.  The card
is filled up with an untouched tensor to just short of what each step needs."""

import numpy as np
import pytest

import polariseq_b200 as pq
from polariseq_b200 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def leave(nbytes):
    """A tensor that leaves about `nbytes` free on the card."""
    import torch

    return torch.empty(free_bytes() - nbytes, dtype=torch.uint8, device="cuda")


def exact(ctx, x, k=10):
    n = len(x)
    ip = np.empty(n + 1, np.uint32)
    ix = np.empty(n * (k - 1), np.uint32)
    dx = np.empty(n * (k - 1), np.float32)
    ctx.neighbors_into(x, k, pq.METRICS["euclidean"], ip, ix, dx)
    return ix.tobytes(), dx.tobytes()


def graph(ctx, x, k=15):
    n = len(x)
    ip = np.empty(n + 1, np.uint32)
    ix = np.empty(n * k, np.uint32)
    dx = np.empty(n * k, np.float32)
    nnz = ctx.nndescent_into(x, pq._opts(k, 2, 0, 0, 0, 0.001), ip, ix, dx)
    return ix[:nnz].tobytes(), dx[:nnz].tobytes()


def test_a_build_takes_the_filters_workspace_back():
    x = synth.mixture_dirichlet(60_000, 20, 8, seed=1)
    y = synth.mixture_dirichlet(400_000, 20, 8, seed=2)
    before = free_bytes()
    ctx = pq.Context(0)
    want = graph(ctx, y)
    need = before - free_bytes()  # what the build keeps (at least; growing takes more)
    ctx.close()
    ctx = pq.Context(0)
    near = exact(ctx, x)          # more than 1 GB of workspace
    ballast = leave(need - 300 * MB)
    try:
        assert graph(ctx, y) == want
    finally:
        del ballast
        free_bytes()
    assert exact(ctx, x) == near  # and the filter gets its workspace again
    ctx.close()


def test_a_set_up_without_room_gives_back_what_it_got():
    x = synth.mixture_dirichlet(60_000, 20, 8, seed=1)
    ctx = pq.Context(0)
    want = exact(ctx, x)
    ctx.close()
    ctx = pq.Context(0)
    exact(ctx, x[:600])            # (kernels loaded, the smallest workspace)
    ballast = leave(500 * MB)      # 1 GB of distances does not fit
    try:
        before = free_bytes()
        assert exact(ctx, x) == want
        # rows, norms and results: 60,000 x (80 + 4 + 80) bytes
        assert before - free_bytes() < 40 * MB
    finally:
        del ballast
        free_bytes()
    ctx.close()


def test_batched_search_without_room():
    import torch

    n, k, d = 200_000, 60, 24
    x = torch.from_numpy(synth.mixture_dirichlet(n, d, 8, seed=3)).cuda()
    off, ks = np.array([0, n // 2, n], np.uint64), np.array([k, k], np.uint32)

    def search(ctx):
        oi = torch.zeros(n * k, dtype=torch.int32, device="cuda")
        od = torch.zeros(n * k, dtype=torch.float32, device="cuda")
        ctx.knn_batched_device(x, off, ks, oi, od)
        torch.cuda.synchronize()
        return oi.cpu().numpy().tobytes(), od.cpu().numpy().tobytes()

    ctx = pq.Context(0)
    want = search(ctx)
    ctx.close()
    ctx = pq.Context(0)
    ballast = leave(260 * MB)  # the results and little else
    try:
        before = free_bytes()
        assert search(ctx) == want
        assert before - free_bytes() < 40 * MB
    finally:
        del ballast
        free_bytes()
    ctx.close()
