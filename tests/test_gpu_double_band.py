"""GPU tests of double calls whose error band holds much of the candidate set (clusters tighter than the
tensor cores' rounding, points far from the origin, points of tiny scale, equal points): their queries
are re-ranked in rounds, or handed to the CUDA-core kernel where that is the cheaper way, and the result
is the CUDA-core kernel's bit for bit either way.

Calls of fewer than 32,768 pairs take that kernel directly: the same rows in slices are the reference.
The sizes sit on both sides of the switch between the re-rank's forms (592 queries), of the list that a
CTA holds (1,024 entries) and of the band limit (a twelfth of the candidates)."""
import numpy as np
import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


def _points(kind, N, d, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    X = torch.rand(N, d, generator=g, device="cuda", dtype=torch.float64)
    if kind == "far":
        X += 1e6
    elif kind == "tiny":
        X *= 1e-20
    elif kind == "equal":
        X = X[:7][torch.arange(N, device="cuda") % 7].contiguous()
    elif kind.startswith("clusters"):
        c = int(kind.split()[1])
        X = X[:c][torch.randint(0, c, (N,), generator=g, device="cuda")]
        X = X + 1e-5 * torch.randn(N, d, generator=g, device="cuda", dtype=torch.float64)
    return X


def _call(X, X2, alpha, beta, D, I):
    G.knn_device(X, X2, alpha, X, X2, beta, D, I)


@pytest.mark.parametrize("kind", ["far", "tiny", "equal", "clusters 3", "clusters 10",
                                  "clusters 14", "clusters 30"])
@pytest.mark.parametrize("n,m,d,k", [(40, 30000, 9, 16), (592, 20000, 20, 50), (593, 20000, 20, 50),
                                     (1500, 16000, 33, 100), (70, 1100, 5, 200)])
def test_same_bits_as_the_cuda_cores(kind, n, m, d, k):
    import torch
    X = _points(kind, n + m, d, 6700 + d)
    X2 = X.square().sum(1)
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.arange(m, m + n, device="cuda", dtype=torch.int32)
    D = torch.full((n, k), float("inf"), device="cuda", dtype=torch.float64)
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    _call(X, X2, alpha, beta, D, I)
    step = max(1, 32767 // m)
    rows = np.arange(0, n, max(1, n // 60))
    for r in rows:
        b = beta[r:r + step].contiguous()
        Ds = torch.full((b.numel(), k), float("inf"), device="cuda", dtype=torch.float64)
        Is = torch.full((b.numel(), k), -1, device="cuda", dtype=torch.int32)
        _call(X, X2, alpha, b, Ds, Is)
        assert torch.equal(Ds, D[r:r + step]), r
        assert torch.equal(Is, I[r:r + step]), r


@pytest.mark.parametrize("n", [30, 593])
def test_merges_into_incoming_rows(n):
    import torch
    m, d, k = 20000, 16, 40
    X = _points("clusters 30", n + 2 * m, d, 6800)
    X2 = X.square().sum(1)
    a1 = torch.arange(m, device="cuda", dtype=torch.int32)
    a2 = torch.arange(m, 2 * m, device="cuda", dtype=torch.int32)
    beta = torch.arange(2 * m, 2 * m + n, device="cuda", dtype=torch.int32)
    D = torch.full((n, k), float("inf"), device="cuda", dtype=torch.float64)
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    _call(X, X2, a1, beta, D, I)
    _call(X, X2, a2, beta, D, I)
    for r in range(0, n, 23):
        Ds = torch.full((1, k), float("inf"), device="cuda", dtype=torch.float64)
        Is = torch.full((1, k), -1, device="cuda", dtype=torch.int32)
        b = beta[r:r + 1].contiguous()
        _call(X, X2, a1, b, Ds, Is)
        _call(X, X2, a2, b, Ds, Is)
        assert torch.equal(Ds, D[r:r + 1]) and torch.equal(Is, I[r:r + 1])
