"""GPU: the native host path does not hold the interpreter lock while a launch waits for room in the queue."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls():
    from sglang_b200.layers.quantization.fp8_kernel import sglang_per_token_group_quant_fp8
    from sglang_b200.layers.quantization.fp8_utils import w8a8_block_fp8_linear
    from sglang_b200.sgl_kernel import silu_and_mul
    x = torch.randn(8, 256, device="cuda").to(torch.bfloat16)
    w, s = torch.zeros(128, 256, device="cuda").to(torch.float8_e4m3fn), torch.ones(1, 2, device="cuda")
    return {"silu_and_mul": lambda: silu_and_mul(x), "quant": lambda: sglang_per_token_group_quant_fp8(x, 128),
            "linear": lambda: w8a8_block_fp8_linear(x, w, [128, 128], s)}


@pytest.mark.parametrize("name", ["silu_and_mul", "quant", "linear"])
def test_other_threads_run_while_a_launch_waits(name):
    call = _calls()[name]
    call()
    torch.cuda.synchronize()
    stop, ticks = threading.Event(), []

    def ticker():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    thread = threading.Thread(target=ticker)
    thread.start()
    try:
        torch.cuda._sleep(1_500_000_000)      # keeps the stream busy for the better part of a second; it ends by itself
        start, longest, when = time.perf_counter(), 0.0, (0.0, 0.0)
        while time.perf_counter() - start < 3.0:
            t0 = time.perf_counter()
            call()
            t1 = time.perf_counter()
            if t1 - t0 > longest:
                longest, when = t1 - t0, (t0, t1)
            if longest > 0.1:
                break
    finally:
        stop.set()
        thread.join()
        torch.cuda.synchronize()
    if longest <= 0.1:
        pytest.skip("the launch queue did not fill")
    during = sum(when[0] < t < when[1] for t in ticks)
    assert during > 0.1 * longest / 0.002, (during, longest)
