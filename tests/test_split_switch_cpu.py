"""CPU: SPLIT_K_MODE = "off" keeps every product off the one-call host path, whose C entry splits k-blocks on its own."""
import pytest
import torch

from sglang_b200 import _lib
from sglang_b200.layers.quantization import fp8_kernel, fp8_utils
from sglang_b200.sgl_kernel import gemm

BLOCK = [128, 128]
W = torch.zeros(128, 256, dtype=torch.float8_e4m3fn)
W_SCALE = torch.ones(1, 2)
X = torch.zeros(16, 256, dtype=torch.bfloat16)
CALLS = {
    "fp32": lambda: fp8_utils.w8a8_block_fp8_linear(X, W, BLOCK, W_SCALE),
    "packed": lambda: fp8_utils.deepgemm_w8a8_block_fp8_linear_with_fallback(X, W, BLOCK, W_SCALE),
    "power-of-two": lambda: fp8_utils.deepgemm_w8a8_block_fp8_linear_with_fallback(X, W, BLOCK, W_SCALE,
                                                                                   weight_scale_ue8m0=True),
    "matmul": lambda: fp8_kernel.w8a8_block_fp8_matmul(W, W, torch.ones(128, 2), W_SCALE, BLOCK, torch.bfloat16),
}


class _Host:
    """Stands in for the native module: records what was called and answers the whole-product calls."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return "one call" if name in ("linear", "matmul") else None
        return call


class _PythonPath(Exception):
    pass


def _reached(*args, **kwargs):
    raise _PythonPath


@pytest.mark.parametrize("name", CALLS)
def test_off_never_reaches_a_splitting_host_call(name, monkeypatch):
    host = _Host()
    monkeypatch.setattr(_lib, "host", lambda: host)
    # the first step of the Python path of each function
    monkeypatch.setattr(fp8_utils, "sglang_per_token_group_quant_fp8", _reached)
    monkeypatch.setattr(fp8_kernel, "launch_dense_mm", _reached)
    assert gemm.SPLIT_K_MODE == "auto" and CALLS[name]() == "one call"
    monkeypatch.setattr(gemm, "SPLIT_K_MODE", "off")
    host.calls.clear()
    with pytest.raises(_PythonPath):
        CALLS[name]()
    assert not host.calls
