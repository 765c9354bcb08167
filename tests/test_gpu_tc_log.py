"""GPU tests of the tensor-core pass's quad logs and their re-rank, against the FP64 oracle.

The epilogue logs groups of four adjacent candidates whole; the re-rank reads a query's logs as one
list (one CTA per query up to 592 queries, one warp each beyond), narrows it by a bisection and
sums each exact distance over four lanes. The sizes sit on those edges: the switch between the two
forms, remainders of the four-lane sum and of a tile, one query, one neighbour, lists of every
register size, and bands that overflow the shared list. `order` sorts the candidates so that a
query's neighbours lie side by side (a quad then holds several of them).

Index sets must be identical; distances are FP64 values rounded to float (half an ulp, 6e-8
relative; assert_close allows 1e-6 and the cancellation near zero)."""
import numpy as np
import pytest

from knn_check import is_maxheap
from rnn_b200 import workloads as W
from test_gpu_tc import _run, assert_close, assert_same_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tf32", "bf16", "bf16x3"])
@pytest.mark.parametrize("shape", [
    (592, 3000, 7, 5, "random"), (593, 3000, 7, 5, "random"), (1, 300, 3, 1, "random"),
    (40, 5000, 13, 256, "random"), (700, 2500, 66, 130, "random"), (130, 257, 64, 32, "random"),
    (129, 40000, 20, 64, "sorted"), (640, 9001, 33, 33, "sorted"), (20, 33, 16, 64, "random")])
def test_quad_log_sets(oracle, mode, shape):
    n, m, d, k, order = shape
    N = m + n + 5
    X = W.gaussian_mixture_table(2000 + d + m, N, d, dtype=np.float32)
    X2 = W.sq_norms(X)
    perm = W.permutation(2001 + m, N)
    alpha, beta = perm[:m].astype(np.int32), perm[m:m + n].astype(np.int32)
    if order == "sorted":  # by mixture component, then along the first axis
        alpha = alpha[np.lexsort((X[alpha, 0], np.round(X[alpha].sum(axis=1))))]
    alpha = np.ascontiguousarray(alpha)
    D, I, _, _ = _run(mode, X, X2, alpha, beta, k, want_C=False)
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta,
                              np.full((n, k), np.inf, dtype=np.float32),
                              np.full((n, k), -1, dtype=np.int32), clamp=True)
    assert is_maxheap(D)
    assert_same_sets(X, X2, beta, I, Ie, De)
    assert_close(np.sort(D.astype(np.float64), axis=1), De)


@pytest.mark.parametrize("mode", ["bf16", "bf16x3"])
def test_wide_band_merges_unsorted_incoming_rows(oracle, mode):
    """Incoming rows in any order (a caller's own heaps), and a latent set whose near-boundary
    distances are dense, so that the band exceeds the shared list and is taken in parts."""
    N, d, n, k = 12000, 128, 700, 64
    X = W.latent_manifold_table(2100, N, d)
    X2 = W.sq_norms(X)
    perm = W.permutation(2101, N)
    beta, a1, a2 = (perm[:n].astype(np.int32), perm[n:6000].astype(np.int32),
                    perm[6000:].astype(np.int32))
    D1, I1, _, _ = _run(mode, X, X2, a1, beta, k, want_C=False)
    mix = W.permutation(2102, k)  # max-heap order is not required of the merge
    D1, I1 = np.ascontiguousarray(D1[:, mix]), np.ascontiguousarray(I1[:, mix])
    D2, I2, _, _ = _run(mode, X, X2, a2, beta, k, D=D1.copy(), I=I1.copy(), want_C=False)
    De, Ie = oracle.knn_exact(k, X, X2, a2, X, X2, beta, D1, I1, clamp=True)
    assert is_maxheap(D2)
    assert_same_sets(X, X2, beta, I2, Ie, De)
