"""GPU test of engines over few reference points: AUTO's probe batch has no more query rows than the
set has points, so that every size can be served."""
import numpy as np
import pytest

from rnn_b200 import serve as S
from rnn_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref", [1, 20, 127, 129, 1023, 1024, 1500, 2047, 2048, 2049])
@pytest.mark.parametrize("mode", [0, 4])
def test_reference_sets_smaller_than_a_probe_batch(oracle, nref, mode):
    import torch
    d, k = 24, 8
    R = W.uniform_table(5000 + nref, nref, d).astype(np.float32)
    R2 = W.sq_norms(R)
    srv = S.Server(torch.from_numpy(R).cuda(), torch.from_numpy(R2).cuda(), mode=mode, max_k=16,
                   heap_budget=16 << 20, slots=2)
    Q = W.uniform_table(5001, 150, d).astype(np.float32)
    rid = srv.submit(Q, k)
    srv.wait(rid, timeout=60)
    D, I = srv.fetch(rid)
    srv.release(rid)
    srv.close()
    X, X2 = np.concatenate([R, Q]), np.concatenate([R2, W.sq_norms(Q)])
    De, Ie = oracle.knn_exact(k, X, X2, np.arange(nref, dtype=np.int32), X, X2,
                              np.arange(nref, nref + 150, dtype=np.int32), clamp=True)
    assert np.array_equal(np.sort(I, axis=1), np.sort(Ie, axis=1))
    Ds, fin = np.sort(D.astype(np.float64), axis=1), np.isfinite(De)
    assert np.array_equal(np.isfinite(Ds), fin)
    assert np.all(np.abs(Ds[fin] - De[fin]) <= 1e-6 * np.abs(De[fin]) + 1e-9)
