"""GPU tests of float calls with candidates at no distance (a NaN or infinite coordinate): every other
query's list is the one without them, in every arithmetic that returns
FP64 distances, on fresh heaps of both start values, in the
batching form and in the serving form. The maxima of the error bound are not finite then, so the
queries have to go to the exact passes; an index out of range is reported as before."""
import ctypes

import numpy as np
import pytest

from rnn_b200 import batch as B
from rnn_b200 import gsknn as G
from rnn_b200 import serve as S
from rnn_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _table(seed, N, d, broken, bad):
    X = W.uniform_table(seed, N, d).astype(np.float32)
    X2 = W.sq_norms(X)
    X[broken, d // 2] = bad
    X2[broken] = bad
    return X, X2


def _check(oracle, X, X2, good, beta, k, D, I):
    De, Ie = oracle.knn_exact(k, X, X2, good, X, X2, beta,
                              np.full((beta.size, k), np.inf, np.float32),
                              np.full((beta.size, k), -1, dtype=np.int32), clamp=True)
    assert np.array_equal(np.sort(I, axis=1), np.sort(Ie, axis=1))
    Ds = np.sort(D.astype(np.float64), axis=1)
    assert np.all(np.abs(Ds - De) <= 1e-6 * De + 1e-9)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("fresh", [np.inf, 1.79e30])
@pytest.mark.parametrize("mode,n,m,d", [
    (0, 300, 5000, 20), (0, 700, 5000, 20), (0, 3100, 33000, 128), (0, 20, 29000, 300),
    (2, 300, 5000, 33), (3, 300, 5000, 64), (4, 700, 5000, 64)])
def test_other_queries_keep_their_lists(oracle, mode, n, m, d, bad, fresh):
    import torch
    k = 10
    broken = np.arange(5, 60, 7)
    X, X2 = _table(6600 + d, n + m, d, broken, bad)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, n + m, dtype=np.int32)
    t = [torch.from_numpy(a).cuda() for a in (X, X2, alpha, beta)]
    D = torch.full((n, k), fresh, device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    G.set_mode(mode)
    try:
        G.knn_device(t[0], t[1], t[2], t[0], t[1], t[3], D, I)
    finally:
        G.set_mode(0)
    rows = np.linspace(0, n - 1, min(n, 60)).astype(int)
    good = np.setdiff1d(alpha, broken).astype(np.int32)
    _check(oracle, X, X2, good, beta[rows], k, D.cpu().numpy()[rows], I.cpu().numpy()[rows])


def test_a_query_at_no_distance_keeps_its_heap_row():
    import torch
    n, m, d, k = 700, 5000, 20, 10
    X, X2 = _table(6610, n + m, d, np.array([5003, 5100]), np.nan)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, n + m, dtype=np.int32)
    t = [torch.from_numpy(a).cuda() for a in (X, X2, alpha, beta)]
    D = torch.full((n, k), 7.5, device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    G.knn_device(t[0], t[1], t[2], t[0], t[1], t[3], D, I)
    D, I = D.cpu().numpy(), I.cpu().numpy()
    for q in (3, 100):
        assert np.all(D[q] == 7.5) and np.all(I[q] == -1)
    assert np.all(I[np.setdiff1d(np.arange(n), [3, 100])] >= 0)


def test_indices_outside_the_table_are_reported():
    import torch
    n, m, d, k = 300, 5000, 20, 10
    X, X2 = _table(6620, n + m, d, np.array([9]), np.nan)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, n + m, dtype=np.int32)
    beta[17] = -4
    t = [torch.from_numpy(a).cuda() for a in (X, X2, alpha, beta)]
    D = torch.full((n, k), np.inf, device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    with pytest.raises(G.GsknnError):
        G.knn_device(t[0], t[1], t[2], t[0], t[1], t[3], D, I)
        torch.cuda.synchronize()
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        if G.lib().gsknn_stream_status(st):
            raise G.GsknnError(G.last_error()[1])


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_batching_form(oracle, bad):
    import torch
    N, d, k, T = 4000, 24, 8, 3
    broken = np.array([3, 700, 3999])
    X, X2 = _table(6630, N, d, np.array([], dtype=int), bad)
    leaves = B.rkdt_leaves(X, T, 200, 800, 3)
    X[broken, 4] = bad
    X2[broken] = bad
    Xd, X2d = torch.from_numpy(X).cuda(), torch.from_numpy(X2).cuda()
    D = torch.full((N, k), np.inf, device="cuda")
    I = torch.full((N, k), -1, device="cuda", dtype=torch.int32)
    job = B.BatchJob(Xd, X2d, D, I, k, trees_per_pass=T, leaf_min=200, shape=3)
    job.run_pass(leaves)
    job.sync()
    job.close()
    D, I = D.cpu().numpy(), I.cpu().numpy()
    mates = [set() for _ in range(N)]
    for l in range(leaves.nleaves):
        p = leaves.pts[leaves.ptr[l]:leaves.ptr[l + 1]]
        for q in p:
            mates[q].update(p.tolist())
    X64 = X.astype(np.float64)
    for q in np.setdiff1d(np.arange(0, N, 37), broken):
        c = np.setdiff1d(np.array(sorted(mates[q])), broken)
        dist = np.maximum(0.0, -2.0 * X64[c] @ X64[q] + X2[c].astype(np.float64)
                          + float(X2[q]))
        want = np.sort(dist)[:k]
        assert np.all(np.isin(I[q], c))
        assert np.all(np.abs(np.sort(D[q].astype(np.float64)) - want) <= 1e-6 * want + 1e-9)


@pytest.mark.parametrize("mode", [0, 4])
def test_serving_form(oracle, mode):
    import torch
    nref, d, k, n = 4000, 32, 8, 200
    broken = np.array([0, 1500, 3999])
    X, X2 = _table(6640, nref + n, d, broken, np.nan)
    srv = S.Server(torch.from_numpy(X[:nref]).cuda(), torch.from_numpy(X2[:nref]).cuda(),
                   mode=mode, max_k=16, heap_budget=16 << 20, slots=2)
    rid = srv.submit(X[nref:], k)
    srv.wait(rid, timeout=60)
    D, I = srv.fetch(rid)
    srv.release(rid)
    srv.close()
    good = np.setdiff1d(np.arange(nref), broken).astype(np.int32)
    _check(oracle, X, X2, good, np.arange(nref, nref + n, dtype=np.int32), k, D, I)
