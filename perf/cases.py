"""Performance cases: the calls a user of the library makes, with their inputs and exact results.

A case is a dict of plain values. `prepare` makes what a program holds before the call (point
tables, norms, index lists, heaps, a batching job or a server), `run` makes one pass through the
public Python API, `work` counts what the pass cannot do without, and `exact` computes the
returned distances in 64 bits with plain torch.

Kinds of call:
  device  `knn_device` on CUDA tensors: float (tensor cores with the exact re-rank), double and
          the 1-norm; a fresh heap per pass, as a program does for a new batch of queries
  host    `sgsknn` / `dgsknn` on numpy arrays: the reference wrapper's calls
  heap    `gsknn_heap` on a library heap with k beyond the fused lists (4-ary header heaps)
  batch   `BatchJob.run_pass`: all nearest neighbours over the leaves of randomized trees
  serve   `Server`: a burst of requests of different m and k against a resident set
"""
from __future__ import annotations

import numpy as np
import torch

from rnn_b200 import batch as B
from rnn_b200 import gsknn as G
from rnn_b200 import serve as S


def _device(name, dtype, data, N, m, n, d, k, metric="l2", same=True):
    c = dict(kind="device", dtype=dtype, data=data, N=N, m=m, n=n, d=d, k=k, metric=metric,
             same=same)
    return dict(c, name=name) if name else c


def _host(name, dtype, data, N, m, n, d, k):
    c = dict(kind="host", dtype=dtype, data=data, N=N, m=m, n=n, d=d, k=k, metric="l2",
             same=True)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a handful of lookups against a small set: the smallest call, latency and launches
        _device("f32 few queries", "float32", "uniform", 4096, 4096, 16, 32, 8),
        # an ordinary float call at odd sizes, queries from a table of their own
        _device("f32 ordinary", "float32", "mixture", 40009, 30011, 2003, 20, 10, same=False),
        # the benchmark's headline call: one large float call
        _device("f32 large d64", "float32", "mixture", 1048576, 262144, 65536, 64, 32),
        # the precision workload: wide rows, dense near-boundary distances, k = 64
        _device("f32 large d256", "float32", "latent", 294912, 262144, 32768, 256, 64),
        # the reference's basic double problem, device-resident
        _device("f64 d32", "float64", "uniform", 8192, 4096, 4096, 32, 16),
        # a larger double call at odd sizes and a longer list
        _device("f64 d100", "float64", "mixture", 60013, 50021, 5003, 100, 50),
        # the 1-norm metric in float
        _device("f32 l1", "float32", "mixture", 131072, 65536, 8192, 64, 32, metric="l1"),
        # the reference wrapper's double call on host arrays
        _host("host f64", "float64", "uniform", 8192, 4096, 4096, 32, 16),
        # a large float call on host arrays: gather, copies, search and copy back
        _host("host f32", "float32", "mixture", 524288, 131072, 16384, 64, 32),
        # double lists beyond the fused kernels, into the library's 4-ary heaps
        dict(name="heap f64 k600", kind="heap", dtype="float64", data="uniform", N=20000,
             m=16384, n=1024, d=32, k=600, metric="l2", same=True),
        # one pass over 8 randomized trees
        dict(name="batch trees", kind="batch", N=262144, d=64, k=32, trees=8, leaf_min=256,
             leaf_max=2048),
        # a burst of mixed requests against a resident set
        dict(name="serve burst", kind="serve", nref=1048576, d=128, requests=24, m_max=4096,
             max_k=64),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    data = rng.choice(["uniform", "mixture", "latent"])
    p = rng.random()
    if p < 0.06:
        leaf_min = rng.randint(128, 512)
        return dict(kind="batch", N=rng.randint(60000, 300000), d=rng.randint(20, 128),
                    k=rng.randint(8, 64), trees=rng.randint(2, 8), leaf_min=leaf_min,
                    leaf_max=leaf_min * rng.randint(3, 8))
    if p < 0.12:
        return dict(kind="serve", nref=_log_int(rng, 100000, 1000000), d=rng.randint(32, 200),
                    requests=rng.randint(8, 24), m_max=rng.choice([512, 1024, 4096]), max_k=64)
    if p < 0.18:
        m = _log_int(rng, 2000, 20000)
        return dict(kind="heap", dtype="float64", data=data, N=m + rng.randint(0, m), m=m,
                    n=_log_int(rng, 32, 1500), d=_log_int(rng, 4, 128),
                    k=rng.randint(513, 1000), metric="l2", same=True)
    if p < 0.32:  # host arrays
        dt = rng.choice(["float32", "float64"])
        top = 130000 if dt == "float32" else 20000
        n, m = _log_int(rng, 16, top // 8), _log_int(rng, 500, top)
        return _host(None, dt, data, max(n, m) + rng.randint(0, 2 * m), m, n,
                     _log_int(rng, 4, 128), _log_int(rng, 1, 64))
    same = rng.random() < 0.6
    if p < 0.55:  # double, or the 1-norm in either precision
        metric = "l1" if p < 0.42 else "l2"
        dt = "float64" if metric == "l2" else rng.choice(["float32", "float64"])
        d = _log_int(rng, 3, 256)
        n, m = _log_int(rng, 1, 8192), _log_int(rng, 300, 65536)
        while n * m * d > 1.7e10:
            n, m = max(1, n // 2), max(300, m * 2 // 3)
        k = min(_log_int(rng, 1, 200), m)
        return _device(None, dt, data, max(n, m) + rng.randint(0, m), m, n, d, k, metric, same)
    d = _log_int(rng, 3, 300)
    n, m = _log_int(rng, 1, 65536), _log_int(rng, 300, 262144)
    while n * m > 4.3e9 or n * m * d > 5e11:
        n, m = max(1, n // 2), max(300, m * 3 // 4)
    k = min(_log_int(rng, 1, 128), m)
    return _device(None, "float32", data, max(n, m) + rng.randint(0, m), m, n, d, k, "l2", same)


# ---- inputs ---------------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFF)
    return g


def _table(data, N, d, dtype, seed, salt):
    """N x d points on the GPU: i.i.d. U[0,1); 16 Gaussians (sigma 0.05) with centres in
    U[0,1)^d; or an 8-dimensional latent cube mapped into R^d with N(0, 1e-3) noise."""
    g = _gen(seed, salt)
    shape = _gen(seed, 1)  # mixture centres and latent basis: one distribution per seed
    if data == "uniform":
        return torch.rand(N, d, generator=g, device="cuda", dtype=dtype)
    if data == "mixture":
        centres = torch.rand(16, d, generator=shape, device="cuda", dtype=dtype)
        label = torch.randint(0, 16, (N,), generator=g, device="cuda")
        X = torch.randn(N, d, generator=g, device="cuda", dtype=dtype)
        return X.mul_(0.05).add_(centres[label])
    r = min(8, d)
    basis, _ = torch.linalg.qr(torch.randn(d, r, generator=shape, device="cuda",
                                           dtype=torch.float64))
    Z = torch.rand(N, r, generator=g, device="cuda", dtype=torch.float64)
    X = (Z @ basis.T).to(dtype)
    return X.add_(torch.randn(N, d, generator=g, device="cuda", dtype=dtype), alpha=1e-3)


def _norms(X):
    return torch.cat([x.double().square().sum(1) for x in X.split(1 << 16)]).to(X.dtype)


def _subset(N, count, seed, salt):
    p = torch.randperm(N, generator=_gen(seed, salt), device="cuda")
    return p[:count].to(torch.int32).contiguous()


def _problem(case, seed):
    """(XA, XA2, alpha, XB, XB2, beta): candidates alpha of XA, queries beta of XB."""
    dt = getattr(torch, case["dtype"])
    XA = _table(case["data"], case["N"], case["d"], dt, seed, 2)
    XA2 = _norms(XA)
    if case["same"]:
        XB, XB2 = XA, XA2
    else:
        XB = _table(case["data"], max(case["n"], case["N"] // 8), case["d"], dt, seed, 3)
        XB2 = _norms(XB)
    return (XA, XA2, _subset(XA.shape[0], case["m"], seed, 4), XB, XB2,
            _subset(XB.shape[0], case["n"], seed, 5))


def _requests(case):
    """(m, k) of every request: m log-uniform in [1, m_max], k of {8, 16, 64}; a case's own."""
    rng = np.random.RandomState(case["nref"] + case["requests"])
    m = np.rint(case["m_max"] ** rng.random_sample(case["requests"])).astype(int)
    k = rng.choice([8, 16, 64], case["requests"])
    return [(int(a), int(b)) for a, b in zip(m, k)]


def _serve_inputs(case, seed):
    R = torch.rand(case["nref"], case["d"], generator=_gen(seed, 2), device="cuda")
    reqs = _requests(case)
    Q = torch.rand(sum(m for m, _ in reqs), case["d"], generator=_gen(seed, 3), device="cuda")
    return R, reqs, Q


def _batch_inputs(case, seed):
    X = _table("mixture", case["N"], case["d"], torch.float32, seed, 2)
    leaves = B.rkdt_leaves(X.cpu().numpy(), case["trees"], case["leaf_min"], case["leaf_max"],
                           seed)
    return X, leaves


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        R, reqs, Q = _serve_inputs(case, seed)
        rows = Q.cpu().numpy().copy()
        parts, at = [], 0
        for m, k in reqs:
            parts.append((np.ascontiguousarray(rows[at:at + m]), k))
            at += m
        return dict(case=case, server=S.Server(R, _norms(R), max_k=case["max_k"]), reqs=parts)
    if kind == "batch":
        X, leaves = _batch_inputs(case, seed)
        k = case["k"]
        D = torch.empty(case["N"], k, device="cuda")
        I = torch.empty(case["N"], k, device="cuda", dtype=torch.int32)
        # the tensor-core shape: its lists are the exact neighbours whatever the machine's timings
        # (the autotuner may settle on a shape with 32-bit distances instead)
        job = B.BatchJob(X, _norms(X), D, I, k, case["trees"], case["leaf_min"], shape=3)
        return dict(case=case, job=job, leaves=leaves, D=D, I=I)
    p = _problem(case, seed)
    n, k = case["n"], case["k"]
    if kind == "device":
        return dict(case=case, p=p, D=torch.empty(n, k, device="cuda", dtype=p[0].dtype),
                    I=torch.empty(n, k, device="cuda", dtype=torch.int32))
    XA, XA2, alpha, XB, XB2, beta = (t.cpu().numpy() for t in p)
    if case["same"]:
        XB, XB2 = XA, XA2
    return dict(case=case, p=(XA, XA2, alpha, XB, XB2, beta))


# ---- one pass -------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "device":
        D, I = state["D"], state["I"]
        D.fill_(float("inf"))
        I.fill_(-1)
        G.knn_device(*state["p"], D, I,
                     metric=G.KNN_1NORM if case["metric"] == "l1" else G.KNN_2NORM)
        return D, I
    if kind == "host":
        XA, XA2, alpha, XB, XB2, beta = state["p"]
        n, k = case["n"], case["k"]
        D = np.full((n, k), np.inf, dtype=XA.dtype)
        I = np.full((n, k), -1, dtype=np.int32)
        f = G.sgsknn if case["dtype"] == "float32" else G.dgsknn
        f(case["d"], k, XB, XB2, beta, XA, XA2, alpha, D, I)
        return D, I
    if kind == "heap":
        heap = G.Heap(case["n"], case["k"])
        G.gsknn_heap(case["k"], *state["p"], heap)
        lo, hi = 3, 3 + case["k"]  # entries behind the 3-slot header
        D, I = heap.D[:, lo:hi].copy(), heap.I[:, lo:hi].copy()
        heap.free()
        return D, I
    if kind == "batch":
        state["D"].fill_(float("inf"))
        state["I"].fill_(-1)
        state["job"].run_pass(state["leaves"])
        return state["D"], state["I"]
    server = state["server"]
    ids = [server.submit(Q, k) for Q, k in state["reqs"]]
    out = []
    for rid in ids:
        server.wait(rid)
        out.append(server.fetch(rid))
        server.release(rid)
    return [a for a, _ in out], [b for _, b in out]


# ---- what a pass cannot do without ------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "serve":
        reqs = _requests(case)
        rows = sum(m for m, _ in reqs)
        kmean = sum(m * k for m, k in reqs) / rows
        evals, pts, size = float(rows) * case["nref"], rows + case["nref"], 4
    elif kind == "batch":
        a, b = case["leaf_min"], case["leaf_max"]
        rows, kmean, size = case["N"], case["k"], 4
        leaf = (a * a + a * b + b * b) / 3 / ((a + b) / 2)  # mean leaf size seen by a point
        evals, pts = case["trees"] * case["N"] * leaf, case["N"]
    else:
        rows, kmean = case["n"], case["k"]
        size = 4 if case["dtype"] == "float32" else 8
        evals, pts = float(case["n"]) * case["m"], case["n"] + case["m"]
    per = 2 * case["d"] + (0 if case.get("metric") == "l1" else 3)
    return {"bytes": float(pts * (case["d"] + 1) * size + rows * kmean * (size + 4)),
            "flops": float(evals * per)}


# ---- the same in 64 bits ------------------------------------------------------------------------
def _dists(Q, Q2, C, C2, metric="l2"):
    if metric == "l1":
        return torch.cdist(Q, C, p=1.0)
    return torch.addmm(C2, Q, C.T, alpha=-2.0).add_(Q2[:, None]).clamp_(min=0.0)


def _top(Q, Q2, C, C2, k, metric="l2"):
    """The k smallest distances of every query row, descending (float64, in row blocks)."""
    Q, Q2, C, C2 = (t.double() for t in (Q, Q2, C, C2))
    rows = max(1, (1 << 28) // C.shape[0])
    return torch.cat([_dists(q, q2, C, C2, metric).topk(k, dim=1, largest=False)[0].flip(1)
                      for q, q2 in zip(Q.split(rows), Q2.split(rows))])


def _exact_batch(case, seed):
    X, leaves = _batch_inputs(case, seed)
    X2 = _norms(X).double()
    X, N, k = X.double(), case["N"], case["k"]
    pts = torch.from_numpy(leaves.pts.astype(np.int64)).cuda()
    D = torch.full((N, k), float("inf"), device="cuda", dtype=torch.float64)
    I = torch.full((N, k), -1, device="cuda", dtype=torch.int64)
    for t in range(case["trees"]):
        nd, ni = torch.full_like(D, float("inf")), torch.full_like(I, -1)
        for l in np.nonzero(leaves.tree == t)[0]:
            p = pts[int(leaves.ptr[l]):int(leaves.ptr[l + 1])]
            kk = min(k, p.numel())
            v, i = _dists(X[p], X2[p], X[p], X2[p]).topk(kk, dim=1, largest=False)
            nd[p, :kk], ni[p, :kk] = v, p[i]
        # union by id: equal ids become neighbours in id order and the second one leaves
        D, I = torch.cat([D, nd], 1), torch.cat([I, ni], 1)
        I, at = I.sort(dim=1)
        D = D.gather(1, at)
        D[:, 1:][(I[:, 1:] == I[:, :-1])] = float("inf")
        D, at = D.topk(k, dim=1, largest=False)
        I = I.gather(1, at)
    return D.flip(1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        R, reqs, Q = _serve_inputs(case, seed)
        R2, out, at = _norms(R), [], 0
        for m, k in reqs:
            q = Q[at:at + m]
            # the library takes a request's norms as 64-bit sums rounded to float
            out.append(_top(q, _norms(q), R, R2, k))
            at += m
        return out, [None] * len(out)
    if kind == "batch":
        return _exact_batch(case, seed), None
    XA, XA2, alpha, XB, XB2, beta = _problem(case, seed)
    a, b = alpha.long(), beta.long()
    D = _top(XB[b], XB2[b], XA[a], XA2[a], case["k"], case["metric"])
    # 4-ary heaps hold the same descending rows behind their header
    return D, None
