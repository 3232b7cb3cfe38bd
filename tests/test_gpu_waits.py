"""GPU: the bounded waits end where they say."""
import ctypes
import os
import subprocess

import pytest
import torch

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
