"""GPU test of the size of the error bound E in split BF16 with the norm column: the column is added
last, so its part |cn|/2 takes the roundings of one MMA (17 additions), not those of all products.

With at most 1,024 candidates the shift is their mean, and the bound can be formed here:
    E = 1.25 [2 (3.2 u^2 + n 2^-23 (1 + u)^2 + 2^-22) |q~| M + 3 2^-24 (CN + |qn'| + 2 |q~| M)
              + (17 2^-23 + 2^-24) CN],   u = 2^-8, n = 3 d_pad + 17
with the last term only where the column fits beside the tiles (k = 16: up to d = 128)
(1% for the roundings upward of its terms). The distances themselves have to lie within it, also
where all of the norm comes from a few far points."""
import numpy as np
import pytest

from rnn_b200 import workloads as W
from test_gpu_tc import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [7, 64, 65, 128, 192])
@pytest.mark.parametrize("data", ["uniform", "mixture", "far points"])
def test_bound_of_the_split_format(d, data):
    m, n, k = 1000, 200, 16
    N = m + n
    if data == "mixture":
        X = W.gaussian_mixture_table(6100 + d, N, d, dtype=np.float32)
    else:
        X = W.uniform_table(6100 + d, N, d).astype(np.float32)
    if data == "far points":
        X[::50] *= 30.0
    X2 = W.sq_norms(X)
    alpha, beta = np.arange(m, dtype=np.int32), np.arange(m, N, dtype=np.int32)
    _, _, C, margin = _run("bf16x3", X, X2, alpha, beta, k)
    Xd = X.astype(np.float64)
    exact = -2.0 * Xd[beta] @ Xd[alpha].T + X2[alpha][None, :].astype(np.float64) \
        + X2[beta][:, None].astype(np.float64)
    E = margin.astype(np.float64) / 2.0
    assert np.all(np.abs(C - exact) <= E[:, None])
    mu = Xd[alpha].mean(0).astype(np.float32).astype(np.float64)
    nrm = np.sqrt(((Xd - mu) ** 2).sum(1))
    eff = X2.astype(np.float64) - 2.0 * Xd @ mu + mu @ mu
    q, M, CN, qn = nrm[beta], nrm[alpha].max(), np.abs(eff[alpha]).max(), np.abs(eff[beta])
    u, terms = 2.0 ** -8, 3 * ((d + 63) // 64 * 64) + 17
    want = 1.25 * (2 * (3.2 * u * u + terms * 2.0 ** -23 * (1 + u) ** 2 + 2.0 ** -22) * q * M
                   + 3 * 2.0 ** -24 * (CN + qn + 2 * q * M)
                   + (17 * 2.0 ** -23 + 2.0 ** -24) * CN * (d <= 128))
    assert np.all(np.abs(E - want) <= 0.01 * want)
