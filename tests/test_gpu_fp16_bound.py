"""GPU test of the error bound of the FP16 form, which AUTO takes for its large calls: the approximate
distance of every (query, candidate) pair lies within the stated E of the FP64 distance, and the lists
are the exact ones. The panels are scaled by a power of two taken from a sample of the candidates:
coordinates beyond its range saturate and small ones flush to zero, which the measured residuals have
to cover, so points of all scales, outliers and queries unlike the candidates are among the cases."""
import ctypes

import numpy as np
import pytest

from rnn_b200 import gsknn as G
from rnn_b200 import workloads as W

pytestmark = pytest.mark.gpu

MODE_FP16 = 5


def _run(X, X2, alpha, beta, k):
    import torch
    L = G.lib()
    f = L.gsknn_tc_distances
    vp, ci, ll = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong
    f.argtypes = [ci, ci, ci, ci, ci, vp, vp, ll, vp, vp, vp, ll, vp, vp, vp, ci, vp, ll, vp, vp]
    t = [torch.from_numpy(a).cuda() for a in (X, X2, alpha, beta)]
    n, m = beta.size, alpha.size
    D = torch.full((n, k), float("inf"), device="cuda")
    I = torch.full((n, k), -1, dtype=torch.int32, device="cuda")
    C = torch.full((n, m), float("nan"), device="cuda")
    margin = torch.zeros(n, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    rc = f(MODE_FP16, m, n, X.shape[1], k, t[0].data_ptr(), t[1].data_ptr(), X.shape[0],
           t[2].data_ptr(), t[0].data_ptr(), t[1].data_ptr(), X.shape[0], t[3].data_ptr(),
           D.data_ptr(), I.data_ptr(), k, C.data_ptr(), m, margin.data_ptr(), st)
    assert rc == 0, G.last_error()
    assert L.gsknn_stream_status(vp(st)) == 0
    return D.cpu().numpy(), I.cpu().numpy(), C.cpu().numpy(), margin.cpu().numpy()


def _points(kind, N, m, d):
    if kind == "mixture":
        return W.gaussian_mixture_table(6900 + d, N, d, dtype=np.float64)
    if kind == "clusters":
        return W.gaussian_mixture_table(6900 + d, N, d, sigma=0.002, dtype=np.float64)
    if kind == "latent":
        return W.latent_manifold_table(6900 + d, N, d, dtype=np.float64)
    X = W.uniform_table(6900 + d, N, d, np.float64)
    if kind == "tiny":
        X *= 1e-9
    elif kind == "large":
        X *= 1e7
    elif kind == "outliers":
        X[1:m:97] *= 1e4
    elif kind == "far queries":
        X[m:] += 50.0
    elif kind == "one wide dimension":
        X[:, d // 3] *= 3e3
    elif kind == "offset":
        X += 300.0
    return X


@pytest.mark.parametrize("d", [3, 64, 100, 128, 200, 256, 300])
@pytest.mark.parametrize("kind", ["uniform", "mixture", "clusters", "latent", "tiny", "large",
                                  "outliers", "far queries", "one wide dimension", "offset"])
def test_distances_within_the_bound(oracle, d, kind):
    m, n, k = 2100, 150, 16
    X = _points(kind, m + n, m, d).astype(np.float32)
    X2 = W.sq_norms(X)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, m + n, dtype=np.int32)
    D, I, C, margin = _run(X, X2, alpha, beta, k)
    X64 = X.astype(np.float64)
    exact = -2.0 * X64[beta] @ X64[alpha].T + X2[alpha].astype(np.float64)[None, :] \
        + X2[beta].astype(np.float64)[:, None]
    E = margin.astype(np.float64) / 2.0
    ratio = np.max(np.abs(C - exact) / E[:, None])
    print(f"max |d' - d| / E = {ratio:.3f} ({kind}, d = {d})")
    assert np.all(np.isfinite(C)) and ratio <= 1.0
    De, Ie = oracle.knn_exact(k, X, X2, alpha, X, X2, beta, np.full((n, k), np.inf, np.float32),
                              np.full((n, k), -1, dtype=np.int32), clamp=True)
    assert np.array_equal(np.sort(I, axis=1), np.sort(Ie, axis=1))
