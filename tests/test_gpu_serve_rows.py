"""GPU tests of serving batches of every row count near a workspace's limit, and of an engine whose
full workspaces do not fit the device memory that is left.

Results are checked against FP64 distances formed here: k-th neighbour distances within float
rounding (1e-6 relative), and every returned id at its own FP64 distance."""
import numpy as np
import pytest

from rnn_b200 import serve as S

pytestmark = pytest.mark.gpu


def _refs(n, d, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    R = torch.rand(n, d, generator=g, device="cuda")
    return R, R.double().square().sum(1).float()


def _check(R, R2, Q, k, D, I):
    import torch
    q = torch.from_numpy(Q).cuda().double()
    q2 = torch.from_numpy((Q.astype(np.float64) ** 2).sum(1).astype(np.float32)).cuda().double()
    full = torch.addmm(R2.double(), q, R.double().T, alpha=-2.0).add_(q2[:, None]).clamp_(min=0.0)
    De = full.topk(k, dim=1, largest=False)[0].cpu().numpy()
    ids = torch.from_numpy(I.astype(np.int64)).cuda()
    own = full.gather(1, ids).cpu().numpy()
    assert all(len(set(r)) == k for r in I.tolist())
    assert np.all(np.abs(np.sort(D, axis=1) - De) <= 1e-6 * De + 1e-9)
    assert np.all(np.abs(own - D) <= 1e-6 * own + 1e-9)


@pytest.mark.parametrize("mode", [0, 4])
def test_row_counts_up_to_the_limit(mode):
    R, R2 = _refs(500000, 64, 1)
    srv = S.Server(R, R2, mode=mode, max_batch_queries=512, max_k=64, heap_budget=64 << 20,
                   slots=2, slice_rows=512)
    rng = np.random.default_rng(2)
    for rows in range(385, 513):
        Q = rng.random((rows, 64), dtype=np.float32)
        k = 64 if rows % 2 else 16
        rid = srv.submit(Q, k)
        srv.wait(rid, timeout=60)
        D, I = srv.fetch(rid)
        srv.release(rid)
        some = rng.integers(0, rows, 8)
        _check(R, R2, Q[some], k, D[some], I[some])
    srv.close()


def test_smaller_workspaces_when_memory_is_short():
    import ctypes
    import torch
    from rnn_b200 import gsknn as G
    R, R2 = _refs(300000, 64, 3)
    L = G.lib()
    L.gsknn_serve_workspace_bytes.restype = ctypes.c_size_t
    need = 3 * L.gsknn_serve_workspace_bytes(300000, 64, 4, 8192, 256, 148)
    L.gsknn_release_workspace()
    torch.cuda.empty_cache()
    # leaves less than the full workspaces, more than what the smaller ones and the panels take
    hold = torch.cuda.mem_get_info()[0] - int(0.75 * need) - (512 << 20)
    keep = torch.empty(hold, dtype=torch.uint8, device="cuda")
    srv = S.Server(R, R2, mode=4, max_batch_queries=8192, max_k=256, heap_budget=64 << 20)
    assert torch.cuda.mem_get_info()[0] < need
    Q = np.random.default_rng(4).random((700, 64), dtype=np.float32)
    rid = srv.submit(Q, 256)
    srv.wait(rid, timeout=60)
    D, I = srv.fetch(rid)
    srv.release(rid)
    srv.close()
    del keep
    torch.cuda.empty_cache()
    _check(R, R2, Q[:32], 256, D[:32], I[:32])
