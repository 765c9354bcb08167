"""The tensor-core form where shared memory is short: sizes whose tiles only fit without the norm
column (long query panels, long lists) or with the last pipeline stage that does, in every format,
against the FP64 oracle; and the sizes just beyond, which each format refuses.

Index sets must be identical; distances are FP64 values rounded to float (half an ulp, 6e-8
relative; assert_close allows 1e-6 and the cancellation near zero)."""
import numpy as np
import pytest

from knn_check import is_maxheap
from rnn_b200 import workloads as W
from test_gpu_tc import _run, assert_close, assert_same_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,d,k", [
    ("tf32", 352, 32), ("tf32", 128, 256), ("tf32", 40, 17), ("bf16", 704, 32),
    ("bf16", 256, 256), ("bf16", 50, 64), ("bf16x3", 256, 64), ("bf16x3", 256, 33),
    ("bf16x3", 192, 128), ("bf16x3", 64, 256)])
def test_tight_tiles_against_oracle(oracle, mode, d, k):
    n, m = 260, 4100
    N = n + m
    X = W.gaussian_mixture_table(3100 + d + k, N, d, dtype=np.float32)
    X2 = W.sq_norms(X)
    perm = W.permutation(3101 + d, N)
    alpha, beta = perm[:m].astype(np.int32), perm[m:].astype(np.int32)
    D, I, _, _ = _run(mode, X, X2, alpha, beta, k, want_C=False)
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta,
                              np.full((n, k), np.inf, dtype=np.float32),
                              np.full((n, k), -1, dtype=np.int32), clamp=True)
    assert is_maxheap(D)
    assert_same_sets(X, X2, beta, I, Ie, De)
    assert_close(np.sort(D.astype(np.float64), axis=1), De)


@pytest.mark.parametrize("mode,d,k", [
    ("tf32", 352, 33), ("tf32", 353, 8), ("bf16", 704, 33), ("bf16", 705, 1),
    ("bf16x3", 256, 65), ("bf16x3", 257, 8), ("bf16x3", 192, 129)])
def test_tiles_that_do_not_fit_are_refused(mode, d, k):
    X = W.uniform_table(3200, 300, d).astype(np.float32)
    X2 = W.sq_norms(X)
    alpha, beta = np.arange(200, dtype=np.int32), np.arange(200, 300, dtype=np.int32)
    with pytest.raises(AssertionError, match="shared memory"):
        _run(mode, X, X2, alpha, beta, k, want_C=False)
