"""GPU tests of double calls through the tensor cores (approximate pass on the centred rows rounded
to the MMA format, exact FP64 distances of the band), against the general path and the FP64 oracle.

The general path for double tables is the CUDA-core kernel; a call takes the tensor cores from
32,768 pairs on, and rows it cannot bound go back to the CUDA-core kernels. Query rows are
independent, so the same problem in slices of fewer pairs is the general path's answer, and the two
have to agree bit for bit: the exact distances come out of the same order of operations, and ties
go to the lower id on both. The cases cover both sides of the line, every list size, remainders of
tiles and of the vector loads, offsets and scales beyond the floats' reach, ties, rows that overflow
every band, NaN and infinite coordinates, norms that are not the points' own, heaps in any order,
and lists shorter than k.

Against the oracle, where points carry no common offset: ids identical, and distances within
2 (d + 4) 2^-53 (|q|^2 + |c|^2), the rounding of two FP64 dot products and their sums."""
import numpy as np
import pytest

from rnn_b200 import gsknn as G
from rnn_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _call(X, X2, alpha, beta, D, I):
    import torch
    dev = torch.device("cuda:0")
    t = [torch.from_numpy(a).to(dev) for a in (X, X2, alpha, beta, D, I)]
    G.knn_device(t[0], t[1], t[2], t[0], t[1], t[3], t[4], t[5])
    return t[4].cpu().numpy(), t[5].cpu().numpy()


def _fresh(n, k):
    return np.full((n, k), np.inf), np.full((n, k), -1, dtype=np.int32)


def _general(X, X2, alpha, beta, D0, I0):
    step = max(1, 32767 // alpha.size)
    parts = [_call(X, X2, alpha, np.ascontiguousarray(beta[i:i + step]), D0[i:i + step].copy(),
                   I0[i:i + step].copy()) for i in range(0, beta.size, step)]
    return np.concatenate([p[0] for p in parts]), np.concatenate([p[1] for p in parts])


def _same(X, X2, alpha, beta, D0, I0):
    assert alpha.size < 32768
    D, I = _call(X, X2, alpha, beta, D0.copy(), I0.copy())
    Dg, Ig = _general(X, X2, alpha, beta, D0, I0)
    assert np.array_equal(I, Ig)
    assert np.array_equal(D, Dg, equal_nan=True)
    return D, I


def _check(oracle, X, X2, alpha, beta, k, D0=None, I0=None):
    if D0 is None:
        D0, I0 = _fresh(beta.size, k)
    D, I = _same(X, X2, alpha, beta, D0, I0)
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta, D0, I0, clamp=True)
    D, I = D[:, ::-1], I[:, ::-1]  # ascending by (distance, id), as the oracle's rows
    scale = np.max(np.abs(X2[beta])) + np.max(np.abs(X2[alpha])) \
        + np.max(np.sum(X[beta] ** 2, axis=1)) + np.max(np.sum(X[alpha] ** 2, axis=1))
    tol = 2.0 * (X.shape[1] + 4) * 2.0 ** -53 * scale
    fin = np.isfinite(De)
    assert np.array_equal(fin, np.isfinite(D))
    assert np.all(np.abs(D[fin] - De[fin]) <= tol)
    assert np.array_equal(I, Ie)


def _split(seed, N, n, m):
    perm = W.permutation(seed, N).astype(np.int32)
    return np.ascontiguousarray(perm[:m]), np.ascontiguousarray(perm[m:m + n])


@pytest.mark.parametrize("shape", [
    (1, 300, 3, 1), (31, 1057, 64, 16), (32, 1024, 64, 16), (700, 2500, 1, 3), (130, 257, 130, 40),
    (593, 3001, 33, 100), (64, 9000, 300, 256), (2000, 4100, 31, 32), (40, 33, 16, 20)])
@pytest.mark.parametrize("offset,scale", [(0.0, 1.0), (1e6, 1.0), (-3e4, 1e-9), (0.0, 1e12)])
def test_shapes_and_scales(oracle, shape, offset, scale):
    n, m, d, k = shape
    X = W.gaussian_mixture_table(3000 + d, n + m, d, dtype=np.float64) * scale + offset * scale
    X2 = W.sq_norms(X)
    alpha, beta = _split(3001, n + m, n, m)
    if offset == 0.0:
        _check(oracle, X, X2, alpha, beta, k)
    else:  # the distances' own rounding decides between near neighbours
        _same(X, X2, alpha, beta, *_fresh(n, k))


@pytest.mark.parametrize("kind", ["integer", "equal", "tiny", "huge", "zero_norms"])
def test_data_that_cannot_be_bounded(oracle, kind):
    n, m, d, k = 300, 2500, 12, 24
    X = W.uniform(3100, (n + m, d))
    if kind == "integer":
        X = np.floor(X * 3.0)
    elif kind == "equal":
        X[:] = X[0]
        X[:7] += 1.0
    elif kind == "tiny":
        X *= 1e-30
    elif kind == "huge":
        X *= 1e60
    X2 = W.sq_norms(X) if kind != "zero_norms" else np.zeros(n + m)
    alpha, beta = _split(3101, n + m, n, m)
    _check(oracle, X, X2, alpha, beta, k)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_rows_leave_the_others_alone(oracle, bad):
    """Candidates with a NaN or infinite coordinate are at no distance: every other query's list is
    the one without them."""
    n, m, d, k = 200, 1500, 20, 10
    X = W.uniform(3200, (n + m, d))
    X2 = W.sq_norms(X)
    alpha, beta = _split(3201, n + m, n, m)
    broken = alpha[5:60:7]
    X[broken, 3] = bad
    X2[broken] = bad
    good = np.ascontiguousarray(np.setdiff1d(alpha, broken).astype(np.int32))
    D, I = _same(X, X2, alpha, beta, *_fresh(n, k))
    De, Ie = oracle.knn_exact(k, X, X2, good, X, X2, beta, *_fresh(n, k), clamp=True)
    assert np.array_equal(I[:, ::-1], Ie)
    assert np.allclose(D[:, ::-1], De, rtol=0, atol=2.0 * (d + 4) * 2.0 ** -53 * 4 * d)


def test_merges_and_early_lists(oracle):
    n, m, d, k = 400, 3000, 40, 30
    X = W.latent_manifold_table(3300, n + 2 * m, d, dtype=np.float64)
    X2 = W.sq_norms(X)
    perm = W.permutation(3301, n + 2 * m).astype(np.int32)
    beta, a1, a2 = (np.ascontiguousarray(perm[:n]), np.ascontiguousarray(perm[n:n + m]),
                    np.ascontiguousarray(perm[n + m:]))
    D1, I1 = _call(X, X2, a1, beta, *_fresh(n, k))
    mix = W.permutation(3302, k)
    D1, I1 = np.ascontiguousarray(D1[:, mix]), np.ascontiguousarray(I1[:, mix])
    _check(oracle, X, X2, a2, beta, k, D1, I1)
    # a heap's own start value (1.79e308) instead of inf, and fewer candidates than k
    D0 = np.full((n, k), 1.79e308)
    D, I = _same(X, X2, np.ascontiguousarray(a1[:k - 4]), beta, D0, _fresh(n, k)[1])
    assert np.all(np.sum(I >= 0, axis=1) == k - 4)
    assert np.all(D[I < 0] == 1.79e308)


def test_index_outside_the_table_is_reported():
    X = W.uniform(3400, (3000, 8))
    X2 = W.sq_norms(X)
    alpha = np.arange(2000, dtype=np.int32)
    beta = np.arange(2000, 2100, dtype=np.int32)
    for a, b in ((7, None), (None, 9)):
        al, be = alpha.copy(), beta.copy()
        if a is not None:
            al[a] = 3000
        if b is not None:
            be[b] = -5
        with pytest.raises(G.GsknnError):
            _call(X, X2, al, be, *_fresh(100, 8))
