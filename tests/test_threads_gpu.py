"""Contexts on several threads at once, with row widths, k and candidate counts
that ask for different amounts of dynamic shared memory from the same kernels: a
kernel's limit is one per device, so no launch may lower another's.  Every
thread's graphs are the ones that a lone context builds."""

import threading

import numpy as np
import pytest

import polariseq_b200 as pq
from polariseq_b200 import synth

pytestmark = pytest.mark.gpu

# (n, d, k, candidates): narrow and wide staged margins and subtrees, the sorted
# rows of extract at k = 5 to 90, the replay's at the same, candidate heaps of any size
JOBS = [(9000, 8, 5, 0), (9000, 93, 45, 0), (12000, 45, 90, 70), (12000, 61, 20, 33)]


def build(ctx, x, k, candidates):
    n = len(x)
    opts = pq._opts(k, 3, 0, candidates, 0, 0.001)
    ip = np.empty(n + 1, np.uint32)
    ix = np.empty(n * k, np.uint32)
    dx = np.empty(n * k, np.float32)
    nnz = ctx.nndescent_into(x, opts, ip, ix, dx)
    return ip.tobytes(), ix[:nnz].tobytes(), dx[:nnz].tobytes()


def test_contexts_on_threads_build_the_same_graphs():
    xs = [synth.mixture_dirichlet(n, d, 8, seed=d) for n, d, _, _ in JOBS]
    ctxs = [pq.Context(0) for _ in JOBS]
    want = [build(c, x, k, m) for c, x, (_, _, k, m) in zip(ctxs, xs, JOBS)]
    wrong = []
    start = threading.Barrier(len(JOBS))

    def work(i):
        try:
            start.wait()
            for _ in range(12):
                if build(ctxs[i], xs[i], JOBS[i][2], JOBS[i][3]) != want[i]:
                    wrong.append(i)
        except Exception as e:  # a device error on one thread fails the test
            wrong.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(len(JOBS))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for c in ctxs:
        c.close()
    assert not wrong, wrong
