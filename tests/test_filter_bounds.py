"""The error bound of the filter's approximate distances (csrc/filter.cu).

On the CPU, in FP64: rows split into two BF16 parts as the operands are, the
three products that the tile kernel forms, with nothing rounded in between; the
parts' error is at most 2^-14 |q||x|, pairs with coordinates at the rounding
ties of BF16 come close to it, and the margin of csrc/filter_plan.cuh covers
this and the sums' error on both sides.  On the GPU, searches of points around
such ties equal the full search's, bit for bit."""

import os
import subprocess

import numpy as np
import pytest

import oracle
import polariseq_b200 as pq

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "polariseq_b200", "csrc")


def bf16(x):
    b = np.ascontiguousarray(x, np.float32).view(np.uint32).astype(np.uint64)
    return ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32)


def parts(x):
    hi = bf16(x)
    return hi.astype(np.float64), bf16(x - hi).astype(np.float64)


def split_errors(q, x):
    """|A - D| of row pairs, over |q||x| and over s^2."""
    (qh, ql), (xh, xl) = parts(q), parts(x)
    q, x = q.astype(np.float64), x.astype(np.float64)
    a = (qh * xh + ql * xh + qh * xl).sum(1) - 0.5 * (x * x).sum(1)
    err = np.abs((q * q).sum(1) - 2 * a - ((q - x) ** 2).sum(1))
    nq, nx = np.linalg.norm(q, axis=1), np.linalg.norm(x, axis=1)
    return err / (nq * nx), err / (nq + np.linalg.norm(q - x, axis=1)) ** 2


def near_ties(rng, n, d):
    """Values within a few FP32 steps of the midpoint of two BF16 numbers, and
    beside it where the second part is rounded by most."""
    base = np.float32(1.0) + np.float32(2 ** -8) * rng.choice([1, 3, 5], (n, d)).astype(np.float32)
    off = rng.choice([0, 1, -1, 2 ** 7, -2 ** 7, 2 ** 6], (n, d)) * 2.0 ** -23
    return ((base + off) * np.exp2(rng.integers(-3, 4, (n, d)))
            * rng.choice([-1, 1], (n, d))).astype(np.float32)


def test_split_error_and_margin(tmp_path):
    rng = np.random.default_rng(5)
    worst_p = worst_s = 0.0
    for d in (1, 2, 3, 7, 30, 62):
        for make in (near_ties, lambda r, n, d: r.normal(size=(n, d)).astype(np.float32),
                     lambda r, n, d: r.standard_cauchy((n, d)).astype(np.float32)):
            q = make(rng, 4000, d)
            for x in (q, make(rng, 4000, d), q * np.float32(1 + 2 ** -10),
                      (q + rng.normal(size=q.shape) * 1e-6).astype(np.float32)):
                p, s = split_errors(q, x)
                worst_p, worst_s = max(worst_p, p.max()), max(worst_s, s.max())
    assert worst_p <= 2 ** -14
    assert worst_s > 5.6e-5  # (the bound is nearly attained)
    src, exe = tmp_path / "m.cpp", tmp_path / "m"
    src.write_text('#include "filter_plan.cuh"\n#include <cstdio>\nint main() { std::printf('
                   '"%.17g %.17g %.17g", double(pq::FILTER_MARGIN), pq::FILTER_ERROR_SPLIT, '
                   'pq::FILTER_ERROR_SUMS); }\n')
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    margin, split, sums = map(float, subprocess.run([str(exe)], capture_output=True, text=True,
                                                    check=True).stdout.split())
    assert split >= 2 ** -14 and sums >= 2.6e-5
    # s of a missed neighbour exceeds the bound's by sqrt(margin) at most
    assert margin >= 2 * (split + sums) * (1 + np.sqrt(margin)) ** 2


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 2, 5])
@pytest.mark.parametrize("spread", [0.3, 0.02, 0.002])
def test_searches_around_rounding_ties(d, spread):
    rng = np.random.default_rng(d)
    n = 4000
    x = near_ties(rng, n, d) + (rng.normal(size=(n, d)) * spread).astype(np.float32)
    x = np.concatenate([x, -x]).astype(np.float32)  # (the centre is near zero)
    for k in (3, 24):
        g = pq.knn_batched([x], [k])[0]
        ref = pq.knn_batched([np.ascontiguousarray(np.pad(x, ((0, 0), (0, 63 - d))))], [k])[0]
        for a, b in zip(g, ref):
            assert a.tobytes() == b.tobytes()
    g = pq.neighbors_dense(x, 15, "euclidean")
    ref = oracle.neighbors_exact(x, 15, "euclidean")
    np.testing.assert_array_equal(g["indices"], ref["indices"])
    assert g["data"].tobytes() == ref["data"].tobytes()
