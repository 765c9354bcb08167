"""CPU tests of the serving form's planner: a slot's workspace is sized once, and every batch that
its limits allow has to fit it, whatever its rows and k (a batch that does not fit fails with every
request in it). Workspaces are sized over whole query tiles, so the row counts between them are the
ones to try: all of the last tiles, and the ends of every tile before."""
import ctypes

import pytest

from rnn_b200 import gsknn as G

SMS = 148
MODES = {"auto": 0, "tf32": 2, "bf16": 3, "bf16x3": 4}


def _bind():
    L = G.lib()
    for f in (L.gsknn_serve_workspace_bytes, L.gsknn_serve_batch_bytes):
        f.restype = ctypes.c_size_t
    return L.gsknn_serve_workspace_bytes, L.gsknn_serve_batch_bytes


def _rows(max_q):
    tail = range(max(1, max_q - 300), max_q + 1)
    ends = (r for t in range(128, max_q, 128) for r in range(t - 8, t + 2))
    return sorted({r for r in (*tail, *ends, 1, 2, 100) if r <= max_q})


@pytest.mark.parametrize("max_q", [256, 500, 512, 1000, 1024, 2048, 3000, 4096, 8192])
@pytest.mark.parametrize("nref,d,max_k,mode", [
    (466392, 124, 64, "auto"), (100000, 32, 64, "auto"), (100000, 32, 64, "bf16x3"),
    (1048576, 128, 64, "auto"), (500000, 64, 64, "bf16"), (300000, 200, 40, "tf32"),
    (3000, 16, 8, "auto"), (700000, 96, 256, "auto")])
def test_every_batch_fits_the_workspace(max_q, nref, d, max_k, mode):
    workspace, batch = _bind()
    m = MODES[mode]
    ws = workspace(nref, d, m, max_q, max_k, SMS)
    assert ws > 0
    for k in sorted({1, 16, 33, max_k - 1, max_k}):
        if k > max_k:
            continue
        over = [r for r in _rows(max_q) if batch(nref, d, m, max_q, max_k, r, k, SMS) > ws]
        assert not over, (k, over[:8], len(over))


def test_arguments_outside_the_limits():
    workspace, batch = _bind()
    assert workspace(0, 64, 0, 1024, 64, SMS) == 0
    assert workspace(1000, 64, 0, 1024, 257, SMS) == 0
    assert batch(1000, 64, 0, 1024, 64, 1025, 64, SMS) == 0
    assert batch(1000, 64, 0, 1024, 64, 10, 65, SMS) == 0
