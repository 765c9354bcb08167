"""GPU tests of AUTO's FP16 form against the FP64 oracle.

Large calls with d > 64 run one scaled FP16 MMA per product; the scale comes from a sample of the
candidates, coordinates beyond its range saturate, small ones flush to zero, and all of that enters
the measured residual of the error bound. The cases sit at the K-chunk edges, use points whose
scale is far from 1, rows far outside the sample's range, queries unlike the candidates, clusters
tight enough to overflow the band (the escalation to split BF16), and double tables.

Index sets must be the oracle's; float results are FP64 values rounded to float (assert_close allows
1e-6 and the cancellation near zero), double ones agree within the rounding of two FP64 dot
products."""
import numpy as np
import pytest

from knn_check import is_maxheap
from rnn_b200 import gsknn as G
from rnn_b200 import workloads as W
from test_gpu_tc import assert_close, assert_same_sets

pytestmark = pytest.mark.gpu


def _call(X, X2, alpha, beta, k):
    import torch
    t = [torch.from_numpy(a).to("cuda:0") for a in (X, X2, alpha, beta)]
    D = torch.full((beta.size, k), float("inf"), device="cuda:0", dtype=t[0].dtype)
    I = torch.full((beta.size, k), -1, device="cuda:0", dtype=torch.int32)
    G.knn_device(t[0], t[1], t[2], t[0], t[1], t[3], D, I)
    return D.cpu().numpy(), I.cpu().numpy()


def _check(oracle, X, alpha, beta, k, scale=1.0):
    X2 = W.sq_norms(X)
    D, I = _call(X, X2, alpha, beta, k)
    n = beta.size
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta, np.full((n, k), np.inf, X.dtype),
                              np.full((n, k), -1, dtype=np.int32), clamp=True)
    assert is_maxheap(D)
    assert_same_sets(X, X2, beta, I, Ie, De)
    if X.dtype == np.float32:
        assert_close(np.sort(D.astype(np.float64), axis=1), De, abs_=1e-9 * scale ** 2)
    else:
        tol = 4.0 * (X.shape[1] + 4) * 2.0 ** -53 * np.max(np.abs(X2))
        assert np.max(np.abs(np.sort(D, axis=1) - De)) <= tol


def _split(seed, N, n, m):
    perm = W.permutation(seed, N).astype(np.int32)
    return np.ascontiguousarray(perm[:m]), np.ascontiguousarray(perm[m:m + n])


# products (queries x candidates x padded d) of at least 1.3e10, or 9e6 candidate entries at d > 256
@pytest.mark.parametrize("d,n,m", [(65, 3100, 33000), (128, 3100, 33000), (129, 2100, 33000),
                                   (256, 1600, 33000), (300, 60, 29000)])
@pytest.mark.parametrize("data", ["uniform", "mixture"])
def test_shapes(oracle, d, n, m, data):
    X = (W.uniform_table(4000 + d, n + m, d, np.float32) if data == "uniform"
         else W.gaussian_mixture_table(4000 + d, n + m, d, dtype=np.float32))
    alpha, beta = _split(4001, n + m, n, m)
    sub = beta if n <= 200 else None
    X2 = W.sq_norms(X)
    if sub is not None:
        _check(oracle, X, alpha, beta, 24)
        return
    # the whole call, checked on 150 of its rows
    D, I = _call(X, X2, alpha, beta, 24)
    rows = W.permutation(4002, n)[:150]
    De, Ie = oracle.knn_exact(24, X, X2, alpha, X, X2, np.ascontiguousarray(beta[rows]),
                              np.full((150, 24), np.inf, np.float32),
                              np.full((150, 24), -1, dtype=np.int32), clamp=True)
    assert is_maxheap(D)
    assert_same_sets(X, X2, beta[rows], I[rows], Ie, De)
    assert_close(np.sort(D[rows].astype(np.float64), axis=1), De)


@pytest.mark.parametrize("kind", ["tiny", "large", "outliers", "far queries", "clusters", "equal"])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_scales(oracle, kind, dtype):
    """60 queries x 29,000 candidates, d = 300 (FP16 by its packed entries)."""
    d, n, m = 300, 60, 29000
    X = W.uniform_table(4100, n + m, d, np.float64)
    alpha, beta = _split(4101, n + m, n, m)
    scale = 1.0
    if kind == "tiny":
        scale = 1e-9
    elif kind == "large":
        scale = 1e7
    elif kind == "outliers":  # far beyond the sampled range: saturate in FP16
        X[alpha[1::97]] *= 1e4
    elif kind == "far queries":
        X[beta] += 50.0
    elif kind == "clusters":
        X = W.gaussian_mixture_table(4102, n + m, d, sigma=0.003, dtype=np.float64)
    elif kind == "equal":
        X[alpha] = X[alpha[0]]
    _check(oracle, (X * scale).astype(dtype), alpha, beta, 20, scale=scale)
