"""GPU test of the batching form's tensor-core shape where the workspace of its full logs does not fit
the device memory that is left: the pass runs with smaller logs, and the lists are the same (exact
distances, ties to the lower id; rows whose log overflows are finished over their whole leaf)."""
import pytest

from rnn_b200 import batch as B
from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


def test_smaller_logs_when_memory_is_short():
    import torch
    N, d, k, T = 262144, 32, 128, 2
    g = torch.Generator(device="cuda")
    g.manual_seed(6400)
    X = torch.rand(N, d, generator=g, device="cuda")
    X2 = X.double().square().sum(1).float()
    leaves = B.rkdt_leaves(X.cpu().numpy(), T, 256, 2048, 5)
    out = []
    for left in (None, 3 << 30):
        D = torch.full((N, k), float("inf"), device="cuda")
        I = torch.full((N, k), -1, device="cuda", dtype=torch.int32)
        job = B.BatchJob(X, X2, D, I, k, trees_per_pass=T, leaf_min=256, shape=3)
        keep = None
        if left:
            G.lib().gsknn_release_workspace()
            torch.cuda.empty_cache()
            keep = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8,
                               device="cuda")
        job.run_pass(leaves)  # full logs: 5.0 GB, smaller ones 1.2 GB
        job.sync()
        job.close()
        del keep
        torch.cuda.empty_cache()
        out.append((D, I))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
