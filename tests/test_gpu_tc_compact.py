"""GPU test of band logs that fill and are compacted: queries in tight clusters, whose candidates
within the error bound outnumber a log's 1,024 entries before the threshold has settled, in one
candidate split (16,384 queries). Between the widths, all queries keep their logs, some overflow to
the brute force, and nearly all do.

A sample of the rows is compared with FP64 distances formed here: the sorted distances within float
rounding (1e-6 relative, and 1e-9 for the cancellation near zero), and every id at its own distance."""
import numpy as np
import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [3, 4])
@pytest.mark.parametrize("sigma", [0.01, 0.0085, 0.0075])
@pytest.mark.parametrize("d,k", [(32, 32), (20, 5), (32, 100)])
def test_full_logs_against_fp64(mode, sigma, d, k):
    import torch
    n, m = 16384, 60000
    g = torch.Generator(device="cuda")
    g.manual_seed(6000 + d + k)
    centres = torch.rand(16, d, generator=g, device="cuda")
    X = torch.randn(m, d, generator=g, device="cuda") * sigma
    X += centres[torch.randint(0, 16, (m,), generator=g, device="cuda")]
    X2 = X.double().square().sum(1).float()
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.randperm(m, generator=g, device="cuda")[:n].to(torch.int32)
    D = torch.full((n, k), float("inf"), device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    G.set_mode(mode)
    try:
        G.knn_device(X, X2, alpha, X, X2, beta, D, I)
    finally:
        G.set_mode(0)
    rows = torch.randperm(n, generator=g, device="cuda")[:200]
    q = beta[rows].long()
    full = torch.addmm(X2.double(), X[q].double(), X.double().T, alpha=-2.0)
    full = full.add_(X2[q].double()[:, None]).clamp_(min=0.0)
    De = full.topk(k, dim=1, largest=False)[0].cpu().numpy()
    own = full.gather(1, I[rows].long()).cpu().numpy()
    Dr = D[rows].cpu().numpy()
    assert all(len(set(r)) == k for r in I[rows].cpu().tolist())
    assert np.all(np.abs(np.sort(Dr, axis=1) - De) <= 1e-6 * De + 1e-9)
    assert np.all(np.abs(own - Dr) <= 1e-6 * own + 1e-9)
