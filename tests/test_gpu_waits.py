"""GPU: the bounded waits end where they say, and time spent behind another kernel does not count against them."""
import ctypes
import os
import subprocess

import pytest
import torch

from oracle import block_fp8_oracle as O

pytestmark = pytest.mark.gpu
LIMIT = 2_000_000_000       # cycles, kWaitLimitCycles
WORDS = 1024                # of the status ring that the device code finds from a slot's address


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    from sglang_b200 import build
    so = str(tmp_path_factory.mktemp("probe") / "wait_probe.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native", "wait_probe.cu")
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "-shared", "-cudart", "shared", "-o", so, src], check=True,
                   capture_output=True)
    lib = ctypes.CDLL(so)
    lib.probe_wait_out.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    lib.probe_early_trigger.argtypes = [ctypes.c_longlong, ctypes.c_void_p]
    return lib


def _wait_out(probe, form, already):
    """(returned, cycles, code in the slot, sticky code) of a wait for a barrier that never completes."""
    buf = torch.zeros(2 * WORDS, dtype=torch.int32, device="cuda")
    first = (-(buf.data_ptr() // 4)) % WORDS            # a ring starts on a multiple of its size
    ring = buf[first:first + WORDS]
    assert ring.data_ptr() % (4 * WORDS) == 0 and ring.numel() == WORDS
    ring[8] = already
    out = torch.zeros(2, dtype=torch.int64, device="cuda")
    assert probe.probe_wait_out(form, ring[8:].data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return int(out[0]), int(out[1]), int(ring[8]), int(ring[0])


@pytest.mark.parametrize("form", [0, 1], ids=["pointer", "shared-address"])
def test_a_wait_that_runs_out(probe, form):
    returned, cycles, slot, sticky = _wait_out(probe, form, 0)
    assert (returned, slot, sticky) == (0, 77, 77)
    assert 0.99 * LIMIT < cycles < 1.2 * LIMIT, cycles


@pytest.mark.parametrize("form", [0, 1], ids=["pointer", "shared-address"])
def test_a_wait_leaves_when_another_wait_of_its_launch_gave_up(probe, form):
    returned, cycles, slot, sticky = _wait_out(probe, form, 5)
    assert (returned, slot, sticky) == (0, 5, 0)        # nothing is reported twice
    assert cycles < 0.25 * LIMIT, cycles


@pytest.mark.parametrize("M,N,K", [(16, 1024, 1024), (256, 1024, 1024), (1024, 1024, 1024)])
@pytest.mark.parametrize("packed", [False, True])
def test_a_busy_predecessor_is_not_a_timeout(probe, M, N, K, packed):
    """A kernel that lets its dependents start and then runs for longer than a wait's limit: the GEMM behind it gives its
    usual result."""
    from sglang_b200 import _lib
    from sglang_b200.layers.quantization.fp8_kernel import (sglang_per_token_group_quant_fp8, w8a8_block_fp8_matmul,
                                                            w8a8_block_fp8_matmul_deepgemm)
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    w, s = O.per_block_quant_mxfp8(torch.randn(N, K, generator=torch.Generator().manual_seed(N)) * 0.02)
    w, s = w.cuda(), s.cuda()
    if packed:
        q, qs = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
        call = lambda: w8a8_block_fp8_matmul_deepgemm(q, w, qs, s, [128, 128], torch.bfloat16, weight_scale_ue8m0=True)
    else:
        q, qs = sglang_per_token_group_quant_fp8(x, 128)
        call = lambda: w8a8_block_fp8_matmul(q, w, qs, s, [128, 128], torch.bfloat16)
    usual = call()
    torch.cuda.synchronize()
    assert probe.probe_early_trigger(LIMIT + LIMIT // 2, torch.cuda.current_stream().cuda_stream) == 0
    behind = call()
    status = ctypes.c_int(0)
    _lib.check("status", _lib.lib().b200_gemm_device_status(ctypes.byref(status)))
    assert status.value == 0
    assert torch.equal(behind, usual)
