"""Host copies through the context's pinned ring (csrc/hostcopy.cu) on the GPU:
the bytes arrive as they are, at the sizes where the ring, its slices and its
chunks (4 MB, six of them, staged from 8 MB on) end unevenly, from and to
pageable and pinned arrays, in several threads with a context each."""

import threading

import numpy as np
import pytest

import polariseq_b200 as pq

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("nbytes", [1, 4096, 8 * MB - 1, 8 * MB, 8 * MB + 5, 12 * MB + 4097,
                                    24 * MB, 24 * MB + 1, 61 * MB + 333])
@pytest.mark.parametrize("pinned", [False, True])
def test_round_trip(nbytes, pinned):
    import torch

    a = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
    if pinned:
        t = torch.from_numpy(a).pin_memory()
        a = t.numpy()
    d = torch.zeros(nbytes + 16, dtype=torch.uint8, device="cuda")
    ctx = pq.default_context(0)
    stream = torch.cuda.current_stream().cuda_stream
    ctx.copy_to_device(d, a, 16, stream)
    assert torch.equal(d[16:].cpu(), torch.from_numpy(a.copy()))
    assert int(d[:16].sum()) == 0
    back = np.zeros(nbytes, np.uint8)
    ctx.copy_to_host(back, d[16:], stream)
    np.testing.assert_array_equal(back, a)


def test_threads_with_their_own_contexts():
    import torch

    bad = []

    def work(i):
        ctx = pq.Context(0)
        try:
            a = np.random.default_rng(i).integers(0, 256, 33 * MB + i, dtype=np.uint8)
            d = torch.empty(a.nbytes, dtype=torch.uint8, device="cuda")
            for _ in range(3):
                ctx.copy_to_device(d, a)
                back = np.zeros(a.nbytes, np.uint8)
                ctx.copy_to_host(back, d)
                if not np.array_equal(back, a):
                    bad.append(i)
        finally:
            ctx.close()

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
