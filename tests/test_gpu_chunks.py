"""GPU tests of calls that run in chunks of heap rows: those whose logs would take more than 16 GB
together, and those whose workspace does not fit the device memory that is left. Rows are independent,
so the results have to be those of the whole call, bit for bit, and an index out of range in any
chunk has to be reported.

Where there is no whole call to compare with, a sample of the rows is checked against FP64 distances
formed here (float rounding, 1e-6 relative, and 1e-9 for the cancellation near zero)."""
import ctypes

import numpy as np
import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


def _problem(n, m, d, k, dtype, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    X = torch.rand(max(n, m), d, generator=g, device="cuda", dtype=dtype)
    X2 = torch.cat([x.double().square().sum(1) for x in X.split(1 << 16)]).to(dtype)
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.arange(n, device="cuda", dtype=torch.int32)
    return X, X2, alpha, beta


def _call(X, X2, alpha, beta, k):
    import torch
    D = torch.full((beta.numel(), k), float("inf"), device="cuda", dtype=X.dtype)
    I = torch.full((beta.numel(), k), -1, device="cuda", dtype=torch.int32)
    G.knn_device(X, X2, alpha, X, X2, beta, D, I)
    return D, I


def _check_rows(X, X2, alpha, beta, k, D, I, rows):
    import torch
    q, c = beta[rows].long(), alpha.long()
    full = torch.addmm(X2[c].double(), X[q].double(), X[c].double().T, alpha=-2.0)
    full = full.add_(X2[q].double()[:, None]).clamp_(min=0.0)
    De = full.topk(k, dim=1, largest=False)[0].cpu().numpy()
    own = full.gather(1, I[rows].long()).cpu().numpy()
    Dr = D[rows].double().cpu().numpy()
    assert np.all(np.abs(np.sort(Dr, axis=1) - De) <= 1e-6 * De + 1e-9)
    assert np.all(np.abs(own - Dr) <= 1e-6 * own + 1e-9)


@pytest.mark.parametrize("n,dtype", [(430001, "float32"), (900000, "float32"), (421000, "float64")])
def test_logs_beyond_the_limit(n, dtype):
    import torch
    m, d, k = 34000, 12, 8
    X, X2, alpha, beta = _problem(n, m, d, k, getattr(torch, dtype), 6300)
    D, I = _call(X, X2, alpha, beta, k)
    assert bool((I >= 0).all())
    rows = torch.cat([torch.arange(3), torch.arange(n - 3, n), torch.randint(0, n, (200,))]).cuda()
    _check_rows(X, X2, alpha, beta, k, D, I, rows)
    # one chunk of the same rows
    Ds, Is = _call(X, X2, alpha, beta[-5000:].contiguous(), k)
    assert torch.equal(D[-5000:], Ds) and torch.equal(I[-5000:], Is)


def test_an_index_out_of_range_in_the_first_chunk_is_reported():
    import torch
    n, m, d, k = 430001, 34000, 12, 8
    X, X2, alpha, beta = _problem(n, m, d, k, torch.float32, 6301)
    beta[7] = n + 5
    D = torch.full((n, k), float("inf"), device="cuda")
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    with pytest.raises(G.GsknnError, match="outside its point table"):
        G.knn_device(X, X2, alpha, X, X2, beta, D, I)
        torch.cuda.synchronize()
        L = G.lib()
        if L.gsknn_stream_status(ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)):
            raise G.GsknnError(G.last_error()[1])


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_a_workspace_that_does_not_fit(dtype):
    import torch
    n, m, d, k = 150000, 60000, 32, 32
    X, X2, alpha, beta = _problem(n, m, d, k, getattr(torch, dtype), 6302)
    Dw, Iw = _call(X, X2, alpha, beta, k)
    torch.cuda.synchronize()
    G.lib().gsknn_release_workspace()
    D = torch.full_like(Dw, float("inf"))
    I = torch.full_like(Iw, -1)
    torch.cuda.empty_cache()
    keep = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    try:
        G.knn_device(X, X2, alpha, X, X2, beta, D, I)  # logs of all rows: 6 GB
        torch.cuda.synchronize()
        held = torch.cuda.mem_get_info()[0]
        D.fill_(float("inf"))
        I.fill_(-1)
        G.knn_device(X, X2, alpha, X, X2, beta, D, I)  # in the same workspace
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] == held
    finally:
        del keep
        torch.cuda.empty_cache()
        G.lib().gsknn_release_workspace()
    assert torch.equal(D, Dw) and torch.equal(I, Iw)
