"""GPU tests of float calls with few queries and bands wider than the list of a CTA (1,024 entries):
the partition bound is tightened by the listed entries first, and what still does not fit is re-ranked in
rounds, whose list has to keep the FP64 distances from one to the next (many neighbours here agree to
float rounding). Clusters whose members lie within the tensor cores' rounding of one another.

Index sets are the FP64 oracle's; distances are FP64 values rounded to float (1e-6 relative, and 1e-9
for the cancellation near zero)."""
import numpy as np
import pytest

from knn_check import is_maxheap
from rnn_b200 import workloads as W
from test_gpu_tc import _run, assert_close, assert_same_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tf32", "bf16", "bf16x3"])
@pytest.mark.parametrize("n,m,d,k,sigma", [
    (5, 40000, 16, 32, 1e-4), (592, 30000, 20, 10, 3e-4), (40, 50000, 33, 100, 1e-3),
    (3, 9000, 8, 256, 1e-5), (200, 40000, 64, 64, 3e-3), (1, 60000, 5, 1, 1e-6)])
def test_bands_beyond_the_list(oracle, mode, n, m, d, k, sigma):
    N = n + m
    rng = np.random.default_rng(7000 + d)
    centres = rng.random((6, d))
    X = (centres[rng.integers(0, 6, N)] + sigma * rng.standard_normal((N, d))).astype(np.float32)
    X2 = W.sq_norms(X)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, N, dtype=np.int32)
    D, I, _, _ = _run(mode, X, X2, alpha, beta, k, want_C=False)
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta, np.full((n, k), np.inf, np.float32),
                              np.full((n, k), -1, dtype=np.int32), clamp=True)
    assert is_maxheap(D)
    Ds = np.sort(D.astype(np.float64), axis=1)
    assert_close(Ds, De)
    # (rows whose k-th and (k+1)-th FP64 distances agree to the sums' rounding have no single set)
    X64, n2 = X.astype(np.float64), X2.astype(np.float64)
    full = np.maximum(0.0, -2.0 * X64[beta] @ X64[alpha].T + n2[alpha][None, :] + n2[beta][:, None])
    part = np.partition(full, k, axis=1)[:, :k + 1]
    top = np.sort(part, axis=1)
    clear = top[:, k] - top[:, k - 1] > 8.0 * d * 2.0 ** -53 * (n2[beta] + n2.max())
    assert n < 40 or clear.sum() >= n // 4
    assert_same_sets(X, X2, beta[clear], I[clear], Ie[clear], De[clear])
