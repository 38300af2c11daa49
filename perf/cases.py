"""The workloads that the speed of this framework is measured on.

Each case is one call that a user makes: the kNN graph of an embedding (the
bit-exact NN-Descent, the tensor-core shortlist forms, the learned
initialisation), the exact search, the per-sample searches and scores of
doublet scoring, and the fuzzy connectivities that consume a graph.  A case
names its path and sizes; ``prepare`` makes its inputs on the GPU from a seed
(the values follow ``polariseq_b200.synth``), ``run`` makes the call.

The package's Python functions take and return NumPy arrays, so the cases of
those functions (``host``) include the copies; the others call the context's
device entry points with torch tensors.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import polariseq_b200 as pq

DEV = "cuda"


def listed():
    return [
        # A small dataset (a few thousand cells) through the drop-in call with
        # its defaults: launches and round trips count.
        dict(name="plain_2700_host", path="nnd", host=True, mode="plain", n=2_700, d=50, k=15, comps=12),
        # The 20,000 x 50 workload of the smoke test and the parity tests.
        dict(name="plain_20k_host", path="nnd", host=True, mode="plain", n=20_000, d=50, k=15, comps=20),
        # An ordinary dataset with another PC count and k = 30, ragged sizes.
        dict(name="plain_171k_k30", path="nnd", host=False, mode="plain", n=171_003, d=30, k=30, comps=40),
        # The benchmark's headline size, bit-exact form: atlas-scale data.
        dict(name="plain_4m", path="nnd", host=False, mode="plain", n=4_000_000, d=50, k=15, comps=60),
        # The same size through the BF16 shortlist form (the benchmark's default).
        dict(name="bf16_4m", path="nnd", host=False, mode="bf16", n=4_000_000, d=50, k=15, comps=60),
        # The E4M3 form at k = 30 from host arrays, ragged sizes and 40 PCs.
        dict(name="fp8_600k_k30_host", path="nnd", host=True, mode="fp8", n=600_011, d=40, k=30, comps=40),
        # Learned initial lists, then the reference's rounds.
        dict(name="learned_1m", path="nnd", host=False, mode="learned", n=1_000_000, d=50, k=15, comps=40),
        # The exact search that small datasets use.
        dict(name="exact_20k_host", path="exact", host=True, metric="euclidean", n=20_000, d=50, k=15, comps=20),
        # The exact search with the cosine metric at its upper sizes, ragged.
        dict(name="exact_60k_cosine", path="exact", host=False, metric="cosine", n=60_013, d=30, k=31, comps=30),
        # Per-sample searches of doublet scoring: uneven samples, cells plus
        # twice as many simulated doublets, k = round(0.5 sqrt(cells)).
        dict(name="batched_24_samples", path="batched", samples=24, lo=2_000, hi=40_000, d=30, ratio=2),
        # Doublet scores of a run of samples (points, searches with larger k, scores).
        dict(name="scrublet_8_samples", path="scrublet", samples=8, lo=1_500, hi=12_000, d=30, ratio=2),
        # Connectivities of a million-cell graph, the step after every graph.
        dict(name="fuzzy_1m", path="fuzzy", n=1_000_000, k=15),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "chosen", "learned", "exact", "batched", "scrublet", "fuzzy"])
    d = rng.choice([20, 30, 37, 40, 50, 50])
    if kind == "plain":
        n = _log(rng, 2_000, 2_500_000)
        k = rng.choice([10, 15, 15, 30]) if n < 500_000 else 15
        return dict(path="nnd", host=n < 300_000, mode="plain", n=n, d=d, k=k, comps=rng.randint(8, 60))
    if kind == "chosen":
        n = _log(rng, 100_000, 4_000_000)
        return dict(path="nnd", host=n < 1_000_000, mode=rng.choice(["bf16", "bf16", "fp8"]), n=n, d=d,
                    k=rng.choice([10, 15, 30]), comps=rng.randint(20, 60))
    if kind == "learned":
        return dict(path="nnd", host=False, mode="learned", n=_log(rng, 300_000, 2_000_000), d=d, k=15,
                    comps=rng.randint(20, 60))
    if kind == "exact":
        n = _log(rng, 1_000, 60_000)
        return dict(path="exact", host=n < 30_000, metric=rng.choice(["euclidean", "cosine"]), n=n, d=d,
                    k=rng.choice([6, 15, 16, 31]), comps=rng.randint(5, 30))
    if kind == "batched":
        return dict(path="batched", samples=rng.randint(2, 24), lo=_log(rng, 500, 3_000),
                    hi=_log(rng, 4_000, 40_000), d=rng.choice([20, 30, 30, 50]), ratio=rng.choice([1, 2, 2]))
    if kind == "scrublet":
        return dict(path="scrublet", samples=rng.randint(1, 8), lo=_log(rng, 800, 2_000),
                    hi=_log(rng, 3_000, 12_000), d=rng.choice([20, 30, 30, 50]), ratio=rng.choice([1, 2, 2]))
    return dict(path="fuzzy", n=_log(rng, 10_000, 1_000_000), k=rng.choice([10, 15, 15, 30]))


# ── inputs ─────────────────────────────────────────────────────────────────


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _mixture(g, n, d, comps, doublets=0.05):
    """Gaussian mixture with log-normal cluster sizes, standard deviations
    j^-0.5, and a share of midpoints of two cells (doublets)."""
    w = torch.exp(torch.randn(comps, generator=g, device=DEV))
    means = 4.0 * torch.randn(comps, d, generator=g, device=DEV)
    lab = torch.multinomial(w, n, replacement=True, generator=g)
    spec = torch.arange(1, d + 1, device=DEV, dtype=torch.float32) ** -0.5
    x = torch.randn(n, d, generator=g, device=DEV)
    x *= spec
    x += means[lab]
    m = int(round(doublets * n))
    if m:
        who = torch.randperm(n, generator=g, device=DEV)[:m]
        a = torch.randint(0, n, (m,), generator=g, device=DEV)
        b = torch.randint(0, n, (m,), generator=g, device=DEV)
        x[who] = 0.5 * (x[a] + x[b])
    return x


def _sizes(case):
    """Cells of each sample: evenly spread over the logarithm, made odd."""
    s, lo, hi = case["samples"], math.log(case["lo"]), math.log(case["hi"])
    return [int(math.exp(lo + (hi - lo) * i / max(s - 1, 1))) | 1 for i in range(s)]


def _k_of(n):
    return int(round(0.5 * math.sqrt(n)))


def _graph(g, n, k):
    """A kNN-like graph: cells on a hidden line in random order, each with k
    distinct neighbours among the 40 (or 3k) nearest, ascending distances."""
    half = max(20, (3 * k) // 2)
    place = torch.randperm(n, generator=g, device=DEV)          # cell at each place
    # one edge pattern for every seed, so that the result's size is the case's
    pick = torch.rand(n, 2 * half, generator=_gen(0), device=DEV).topk(k, dim=1).indices
    off = torch.where(pick < half, pick - half, pick - half + 1)
    nbr = place[(torch.arange(n, device=DEV)[:, None] + off) % n]
    # distances of a high-dimensional neighbourhood crowd towards the k-th
    dist = ((torch.arange(k, device=DEV) + torch.rand(n, k, generator=g, device=DEV)) / k) ** 0.2 * 3.0 + 0.2
    dist *= torch.exp(0.3 * torch.randn(n, 1, generator=g, device=DEV))
    idx = torch.empty(n, k, dtype=torch.int64, device=DEV)
    dst = torch.empty(n, k, device=DEV)
    idx[place] = nbr
    dst[place] = dist.sort(1).values
    return idx, dst


def _nnd_opts(case):
    mode = case["mode"]
    kw = dict(init=pq.INITS["learned"]) if mode == "learned" else {}
    return pq._opts(case["k"], 0, 0, 0, 0, 0.001, mode=pq.MODES["plain" if mode == "learned" else mode], **kw)


def _scrublet_inputs(case, seed):
    g = _gen(seed)
    u, w, totals, mv, pairs, ks = [], [], [], [], [], []
    for n in _sizes(case):
        x = _mixture(g, n, case["d"], 10, 0.0).double()
        t = torch.exp(8.0 + 0.4 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64))
        # projected counts of a cell grow with its total: the scaled points keep the mixture
        u.append((x * (t / 1e6)[:, None]).cpu().numpy())
        w.append((1e6 / t).cpu().numpy())
        totals.append(t.cpu().numpy())
        mv.append(x.mean(0).cpu().numpy())
        pairs.append(torch.randint(0, n, (case["ratio"] * n, 2), generator=g, device=DEV).cpu().numpy()
                     .astype(np.uint32))
        ks.append(_k_of(n))
    return u, w, totals, mv, pairs, ks


def prepare(case, seed):
    path = case["path"]
    if path in ("nnd", "exact"):
        x = _mixture(_gen(seed), case["n"], case["d"], case["comps"])
        st = dict(case=case, x=x.cpu().numpy() if case["host"] else x)
        if not case["host"]:
            n, k = case["n"], case["k"]
            per = pq.effective_k(n, k) if path == "nnd" else min(k, n) - 1
            st["ctx"] = pq.default_context()
            st["indptr"] = torch.empty(n + 1, dtype=torch.int32, device=DEV)
            st["indices"] = torch.empty(n * per, dtype=torch.int32, device=DEV)
            st["data"] = torch.empty(n * per, dtype=torch.float32, device=DEV)
            if path == "nnd":
                st["opts"] = _nnd_opts(case)
        return st
    if path == "batched":
        g = _gen(seed)
        samples = []
        for n in _sizes(case):
            x = _mixture(g, n, case["d"], 10, 0.0)
            m = case["ratio"] * n
            a = torch.randint(0, n, (m,), generator=g, device=DEV)
            b = torch.randint(0, n, (m,), generator=g, device=DEV)
            samples.append(torch.cat([x, 0.5 * (x[a] + x[b])]).cpu().numpy())
        return dict(case=case, samples=samples, ks=[_k_of(n) for n in _sizes(case)])
    if path == "scrublet":
        return dict(case=case, inputs=_scrublet_inputs(case, seed))
    idx, dst = _graph(_gen(seed), case["n"], case["k"])
    n, k = case["n"], case["k"]
    return dict(case=case, indptr=np.arange(n + 1, dtype=np.uint32) * np.uint32(k),
                indices=idx.reshape(-1).cpu().numpy().astype(np.uint32), data=dst.reshape(-1).cpu().numpy())


# ── the calls ──────────────────────────────────────────────────────────────


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "nnd":
        if case["host"]:
            mode = case["mode"]
            if mode == "learned":
                g = pq.nndescent_dense(state["x"], case["k"], init="learned")
            else:
                g = pq.nndescent_dense(state["x"], case["k"], mode=mode)
            return {"indptr": g["indptr"], "indices": g["indices"], "data": g["data"]}
        nnz = state["ctx"].nndescent_device(state["x"], state["opts"], state["indptr"], state["indices"],
                                            state["data"])
        return {"indptr": state["indptr"], "indices": state["indices"][:nnz], "data": state["data"][:nnz]}
    if path == "exact":
        if case["host"]:
            g = pq.neighbors_dense(state["x"], case["k"], case["metric"])
            return {"indptr": g["indptr"], "indices": g["indices"], "data": g["data"]}
        nnz = state["ctx"].neighbors_device(state["x"], case["k"], pq.METRICS[case["metric"]], state["indptr"],
                                            state["indices"], state["data"])
        return {"indptr": state["indptr"], "indices": state["indices"][:nnz], "data": state["data"][:nnz]}
    if path == "batched":
        return pq.knn_batched(state["samples"], state["ks"])
    if path == "scrublet":
        u, w, totals, mv, pairs, ks = state["inputs"]
        return pq.scrublet_scores(u, w, totals, mv, pairs, ks, 0.08)
    g = pq.fuzzy_connectivities(state["indptr"], state["indices"], state["data"], case["n"])
    return {"indptr": g["indptr"], "indices": g["indices"], "data": g["data"]}


def work(case):
    """Inputs read once, outputs written once; a search's operations are one
    distance (subtract, multiply, add per dimension) per pair of points, a
    graph's one per neighbour."""
    path = case["path"]
    if path == "nnd":
        n, d, k = case["n"], case["d"], case["k"]
        return {"bytes": 4 * (n * d + 2 * n * k + n + 1), "flops": 3 * d * n * k}
    if path == "exact":
        n, d, k = case["n"], case["d"], case["k"]
        return {"bytes": 4 * (n * d + 2 * n * (k - 1) + n + 1), "flops": 3 * d * n * (n - 1) / 2}
    if path in ("batched", "scrublet"):
        byts = flops = 0
        for n in _sizes(case):
            pts, k = (1 + case["ratio"]) * n, _k_of(n)
            flops += 3 * case["d"] * pts * (pts - 1) / 2
            byts += pts * case["d"] * 4 + 8 * pts * k if path == "batched" else 8 * (n * case["d"] + 2 * n + 2 * pts)
        return {"bytes": byts, "flops": flops}
    n, k = case["n"], case["k"]
    return {"bytes": 4 * (2 * n + 2 + 2 * n * k + 2 * 1.5 * n * k), "flops": 20 * n * k}


# ── the same in 64 bits ────────────────────────────────────────────────────


def _nearest64(x, k, cosine=False, drop_self=True):
    """Ascending distances of each row's k nearest (other) rows."""
    n = x.shape[0]
    if cosine:
        x = x / x.norm(dim=1, keepdim=True)
    sq = (x * x).sum(1)
    out = torch.empty(n, k, dtype=torch.float64, device=x.device)
    idx = torch.empty(n, k, dtype=torch.int64, device=x.device)
    step = max(1, (1 << 28) // max(n, 1))
    for s in range(0, n, step):
        e = min(n, s + step)
        dt = x[s:e] @ x.T
        dd = 1.0 - dt if cosine else (sq[s:e, None] + sq[None, :] - 2.0 * dt).clamp_(min=0.0)
        if drop_self:
            dd[torch.arange(e - s, device=x.device), torch.arange(s, e, device=x.device)] = math.inf
        v, i = dd.topk(k, dim=1, largest=False)
        out[s:e] = v if cosine else v.sqrt()
        idx[s:e] = i
    return out, idx


def _scrublet64(case, seed):
    u, w, totals, mv, pairs, ks = _scrublet_inputs(case, seed)
    out = []
    for uu, ww, tt, m, pr, k in zip(u, w, totals, mv, pairs, ks):
        uu, ww, tt, m = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in (uu, ww, tt, m))
        a, b = (torch.from_numpy(pr[:, j].astype(np.int64)).to(DEV) for j in (0, 1))
        pts = torch.cat([ww[:, None] * uu - m, (1e6 / (tt[a] + tt[b]))[:, None] * (uu[a] + uu[b]) - m])
        n, r = uu.shape[0], pr.shape[0] / uu.shape[0]
        kadj = min(max(int(np.round(k * (1 + r))), 1), pts.shape[0] - 1)
        _, idx = _nearest64(pts.float().double(), kadj)
        q = ((idx >= n).sum(1).double() + 1.0) / (kadj + 2.0)
        rho = 0.08
        sc = q * rho / r / ((1 - rho) - q * (1 - rho - rho / r))
        out.append({"obs": sc[:n], "sim": sc[n:], "k_adj": None})
    return out


def _fuzzy64(case, seed):
    idx, dst = _graph(_gen(seed), case["n"], case["k"])
    n, k = idx.shape
    d = dst.double()
    rho = d[:, :1]
    target = math.log2(k + 1)
    lo, hi = torch.zeros(n, 1, device=DEV).double(), torch.full((n, 1), math.inf, device=DEV).double()
    mid, done = torch.ones(n, 1, device=DEV).double(), torch.zeros(n, 1, device=DEV, dtype=torch.bool)
    for _ in range(64):
        s = torch.where(d > rho, torch.exp(-(d - rho) / mid), 1.0).sum(1, keepdim=True)
        done |= (s - target).abs() < 1e-5
        up = s > target
        hi = torch.where(~done & up, mid, hi)
        lo = torch.where(~done & ~up, mid, lo)
        mid = torch.where(done, mid, torch.where(hi.isinf(), mid * 2, (lo + hi) / 2))
    sigma = torch.maximum(mid, 1e-3 * d.sum(1, keepdim=True) / (k + 1))
    wt = torch.where(d > rho, torch.exp(-(d - rho) / sigma), 1.0).reshape(-1)
    row, col = torch.arange(n, device=DEV).repeat_interleave(k), idx.reshape(-1)
    key = torch.cat([row * n + col, col * n + row])
    uniq, inv = key.unique(return_inverse=True)
    total = torch.zeros(uniq.numel(), device=DEV).double().index_add_(0, inv, torch.cat([wt, wt]))
    keep = torch.ones_like(total).index_reduce_(0, inv, torch.cat([wt, wt]), "prod")
    count = torch.zeros(uniq.numel(), device=DEV).double().index_add_(0, inv, torch.ones(key.numel(), device=DEV).double())
    val = torch.where(count > 1, total - keep, total)
    return {"indptr": None, "indices": None, "data": val[val > 1e-5]}


def exact(case, seed):
    path = case["path"]
    if path == "exact":
        x = _mixture(_gen(seed), case["n"], case["d"], case["comps"]).double()
        v, _ = _nearest64(x, min(case["k"], case["n"]) - 1, case["metric"] == "cosine")
        return {"indptr": None, "indices": None, "data": v.reshape(-1)}
    if path == "batched":
        st = prepare(case, seed)
        return [(None, _nearest64(torch.from_numpy(s).to(DEV).double(), k)[0])
                for s, k in zip(st["samples"], st["ks"])]
    if path == "scrublet":
        return _scrublet64(case, seed)
    if path == "fuzzy":
        return _fuzzy64(case, seed)
    return None  # an approximate graph has no value apart from its search
