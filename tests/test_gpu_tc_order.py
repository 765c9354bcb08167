"""GPU test of one order of summation: a query's distances are the same bits whether its band fitted
its logs (re-rank, by warps or by CTAs) or overflowed them (brute force). The same queries run in calls
of 16,384 rows (one candidate split, whose logs clusters overflow), 700 and 100 rows (many splits, whose
logs hold every candidate)."""
import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 7, 16, 19, 20, 32, 45, 64])
def test_same_bits_on_every_path(d):
    import torch
    n, m, k = 16384, 33000, 64
    g = torch.Generator(device="cuda")
    g.manual_seed(6500 + d)
    # values of 24 significant bits with widely different exponents: sums that round
    X = torch.randn(m, d, generator=g, device="cuda") * 1e-4
    X += torch.rand(8, d, generator=g, device="cuda")[torch.randint(0, 8, (m,), generator=g,
                                                                    device="cuda")]
    X2 = X.double().square().sum(1).float()
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.randperm(m, generator=g, device="cuda")[:n].to(torch.int32)

    def call(rows):
        b = beta[:rows].contiguous()
        D = torch.full((rows, k), float("inf"), device="cuda")
        I = torch.full((rows, k), -1, device="cuda", dtype=torch.int32)
        G.knn_device(X, X2, alpha, X, X2, b, D, I)
        return D, I

    D, I = call(n)
    for rows in (700, 100):
        Dr, Ir = call(rows)
        assert torch.equal(Dr, D[:rows])
        assert torch.equal(Ir, I[:rows])
