"""GPU test of the brute-force pass behind the tensor-core form: clusters so tight that every query's
band overflows its logs (16,384 queries, one candidate split), at every remainder of the dot product's
four-dimension groups and with rows that are and are not 16-byte aligned.

A sample of the rows is compared with FP64 distances formed here: the sorted distances within float
rounding (1e-6 relative, and 1e-9 for the cancellation near zero), and every id at its own distance."""

import numpy as np
import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,k", [(1, 3), (3, 32), (4, 33), (5, 1), (30, 8), (31, 100), (33, 16),
                                 (64, 32), (127, 5)])
def test_all_rows_against_fp64(d, k):
    import torch
    n, m = 16384, 33000
    g = torch.Generator(device="cuda")
    g.manual_seed(6200 + d)
    centres = torch.rand(8, d, generator=g, device="cuda")
    X = torch.randn(m, d, generator=g, device="cuda") * 1e-4
    X += centres[torch.randint(0, 8, (m,), generator=g, device="cuda")]
    X2 = X.double().square().sum(1).float()
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.randperm(m, generator=g, device="cuda")[:n].to(torch.int32)
    D = torch.full((n, k), float("inf"), device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    G.knn_device(X, X2, alpha, X, X2, beta, D, I)
    rows = torch.randperm(n, generator=g, device="cuda")[:100]
    q = beta[rows].long()
    full = torch.addmm(X2.double(), X[q].double(), X.double().T, alpha=-2.0)
    full = full.add_(X2[q].double()[:, None]).clamp_(min=0.0)
    De = full.topk(k, dim=1, largest=False)[0].cpu().numpy()
    own = full.gather(1, I[rows].long()).cpu().numpy()
    Dr = D[rows].cpu().numpy()
    assert all(len(set(r)) == k for r in I[rows].cpu().tolist())
    assert np.all(np.abs(np.sort(Dr, axis=1) - De) <= 1e-6 * De + 1e-9)
    assert np.all(np.abs(own - Dr) <= 1e-6 * own + 1e-9)
