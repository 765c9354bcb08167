"""GPU test of the arithmetic AUTO takes for large float calls, by the bits of its results' band: below
d = 128 a call in AUTO and one in split BF16 launch the same kernels (no escalation pass), from d = 128
AUTO runs FP16 with its escalation behind it."""
import ctypes
import json

import pytest

from rnn_b200 import gsknn as G

pytestmark = pytest.mark.gpu


def _kernels(mode, d, dtype):
    import torch
    n, m, k = 3100, 36000, 16  # at least 1.3e10 products from d = 65 on
    g = torch.Generator(device="cuda")
    g.manual_seed(d)
    X = torch.rand(n + m, d, generator=g, device="cuda", dtype=getattr(torch, dtype))
    X2 = X.double().square().sum(1).to(X.dtype)
    alpha = torch.arange(m, device="cuda", dtype=torch.int32)
    beta = torch.arange(m, m + n, device="cuda", dtype=torch.int32)
    D = torch.full((n, k), float("inf"), device="cuda", dtype=X.dtype)
    I = torch.full((n, k), -1, device="cuda", dtype=torch.int32)
    L = G.lib()
    buf = ctypes.create_string_buffer(1 << 16)
    G.set_mode(mode)
    L.gsknn_trace_enable(1)
    try:
        G.knn_device(X, X2, alpha, X, X2, beta, D, I)
        torch.cuda.synchronize()
        L.gsknn_trace_read(buf, len(buf))
    finally:
        L.gsknn_trace_enable(0)
        G.set_mode(0)
    return {name: v["launches"] for name, v in json.loads(buf.value).items()}


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("d,escalates", [(65, False), (100, False), (127, False), (128, True),
                                         (192, True)])
def test_large_calls_take_fp16_from_d_128(d, escalates, dtype):
    auto = _kernels(0, d, dtype)
    assert ("tc_escalate" in auto) == escalates
    if dtype == "float32" and not escalates:
        assert auto == _kernels(4, d, dtype)


def test_the_cuda_core_mode_holds_for_doubles():
    """GSKNN_MODE_FP32 keeps double calls on the CUDA-core kernels, with the same results."""
    auto, cores = _kernels(0, 20, "float64"), _kernels(1, 20, "float64")
    assert "tc_knn" in auto
    assert "fused_knn_simt" in cores and not any(name.startswith("tc_") for name in cores)
