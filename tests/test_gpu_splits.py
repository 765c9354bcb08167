"""Candidate splits of the CUDA-core kernels: calls whose split count lies at the ends of its
range (every slot for few queries, one or two splits for many) and calls with a last split that
is short, 1-norm and FP32-mode 2-norm, float and double.

The 1-norm is a sum in dimension order in the input precision and ties go to the lower id, so
heaps equal the oracle's bit for bit whatever the split. The FP32-mode 2-norm does not depend on
the split either: a distance is one dot product whose order the tile fixes, so the heap over all
candidates equals, bit for bit, one that is built over slices of the candidates (which take
other split counts).
"""
import numpy as np
import pytest

from knn_check import is_maxheap, sorted_rows
from rnn_b200 import gsknn as G
from rnn_b200 import workloads as W

pytestmark = pytest.mark.gpu

SHAPES = [(1, 30011, 5, 16), (3, 40000, 9, 64), (3, 40000, 9, 65), (129, 2500, 33, 200),
          (5000, 1500, 7, 100), (20000, 300, 4, 64), (6000, 129, 3, 33)]


def _inputs(n, m, d, k, dtype):
    N = n + m
    X = W.uniform_table(900 + k, N, d).astype(dtype)
    p = W.permutation(901 + k, N).astype(np.int32)
    return X, p[:m], p[m:]


def _run(torch, Xt, x2, alpha, beta, k, metric):
    D = torch.full((beta.size, k), float("inf"), dtype=Xt.dtype, device="cuda")
    I = torch.full((beta.size, k), -1, dtype=torch.int32, device="cuda")
    bt = torch.from_numpy(beta).cuda()
    for a in alpha:
        G.knn_device(Xt, x2, torch.from_numpy(a).cuda(), Xt, x2, bt, D, I, metric=metric)
    return sorted_rows(D.cpu().numpy(), I.cpu().numpy()), D.cpu().numpy()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,m,d,k", SHAPES)
def test_l1_does_not_depend_on_the_split(oracle, n, m, d, k, dtype):
    torch = pytest.importorskip("torch")
    X, alpha, beta = _inputs(n, m, d, k, dtype)
    (Ds, Is), D = _run(torch, torch.from_numpy(X).cuda(), None, [alpha], beta, k, G.KNN_1NORM)
    assert is_maxheap(D)
    rows = np.linspace(0, n - 1, min(n, 200)).astype(int)
    De, Ie = oracle.knn_exact_l1(k, X, alpha, X, beta[rows])
    assert np.array_equal(Ds[rows].astype(np.float64), De)
    assert np.array_equal(Is[rows], Ie)


@pytest.mark.parametrize("n,m,d,k", SHAPES)
def test_l2_fp32_does_not_depend_on_the_split(n, m, d, k):
    torch = pytest.importorskip("torch")
    X, alpha, beta = _inputs(n, m, d, k, np.float32)
    Xt = torch.from_numpy(X).cuda()
    x2 = torch.from_numpy(W.sq_norms(X)).cuda()
    G.set_mode(G.MODE_FP32)
    try:
        whole, D = _run(torch, Xt, x2, [alpha], beta, k, G.KNN_2NORM)
        parts, _ = _run(torch, Xt, x2, np.array_split(alpha, 3), beta, k, G.KNN_2NORM)
    finally:
        G.set_mode(G.MODE_AUTO)
    assert is_maxheap(D)
    assert np.array_equal(whole[0], parts[0]) and np.array_equal(whole[1], parts[1])
