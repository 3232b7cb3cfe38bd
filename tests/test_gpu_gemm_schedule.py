"""GPU: the 128-row-tile GEMM at the edges of its tile-width and split rules, against the fp32 oracle product."""
import pytest
import torch

from oracle import block_fp8_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [193, 255, 257, 513])
@pytest.mark.parametrize("N,K", [(576, 4096), (384, 4224), (1280, 640), (2816, 2176)])
@pytest.mark.parametrize("column_major", [False, True])
def test_tile_width_and_split_edges(M, N, K, column_major):
    """Few tiles (split over idle SMs), one 128-column remainder, ragged N; row-major and column-major scales."""
    from sglang_b200.layers.quantization.fp8_kernel import w8a8_block_fp8_matmul
    g = torch.Generator().manual_seed(M + N + K)
    a = (torch.randn(M, K, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    b = (torch.randn(N, K, generator=g) * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    sa, sb = torch.rand(M, K // 128, generator=g) * 0.01, torch.rand((N + 127) // 128, K // 128, generator=g) * 0.01
    sa_d = sa.cuda().t().contiguous().t() if column_major else sa.cuda()
    out = w8a8_block_fp8_matmul(a.cuda(), b.cuda(), sa_d, sb.cuda(), [128, 128], torch.float32).cpu()
    assert O.rel_l2(out, O.block_fp8_matmul_fp32(a, b, sa, sb)) <= 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M", [1, 64, 200])
def test_linear_bias_is_added_to_the_rounded_product(M, dtype):
    from sglang_b200.layers.quantization.fp8_utils import w8a8_block_fp8_linear
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, 1024, generator=g).to(dtype).cuda()
    wq, ws = O.gen_weight(640, 1024, seed=3)
    bias = torch.randn(640, generator=g).to(dtype).cuda()
    plain = w8a8_block_fp8_linear(x, wq.cuda(), [128, 128], ws.cuda())
    with_bias = w8a8_block_fp8_linear(x, wq.cuda(), [128, 128], ws.cuda(), bias=bias)
    plain += bias
    assert torch.equal(plain, with_bias)


@pytest.mark.parametrize("M,N,K", [(16, 7168, 8192), (129, 7168, 8192), (1021, 576, 7168), (1300, 4040, 5248), (64, 128, 128)])
def test_plan_is_what_the_library_runs(M, N, K):
    """The plan's workspace is the one that the automatic schedule uses: the workspace entry point gives the same figure,
    with it the result has the bits of the torch-facing call, and nothing is written beyond it."""
    import ctypes
    from sglang_b200 import _lib
    from sglang_b200.layers.quantization.fp8_kernel import w8a8_block_fp8_matmul
    L = _lib.lib()
    split, nbytes = ctypes.c_int(0), ctypes.c_size_t(0)
    _lib.check("plan", L.b200_fp8_blockwise_scaled_mm_splitk_plan(M, N, K, L.b200_sm_count(), ctypes.byref(split), ctypes.byref(nbytes)))
    assert nbytes.value == L.b200_fp8_blockwise_scaled_mm_workspace_bytes(M, N, K)
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = (torch.randn(M, K, generator=g, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    b = (torch.randn(N, K, generator=g, device="cuda") * 60).clamp(-448, 448).to(torch.float8_e4m3fn)
    sa = torch.rand(M, K // 128, generator=g, device="cuda") * 0.01
    sb = torch.rand((N + 127) // 128, K // 128, generator=g, device="cuda") * 0.01
    out = torch.empty(M, N, device="cuda")
    n = nbytes.value // 4
    ws = torch.full((n + 1024,), 123.0, device="cuda")
    _lib.check("mm", L.b200_fp8_blockwise_scaled_mm_splitk(
        a.data_ptr(), K, b.data_ptr(), K, sa.data_ptr(), K // 128, 1, sb.data_ptr(), K // 128, 1, out.data_ptr(), N,
        _lib.DT_F32, M, N, K, 0, ws.data_ptr() if n else None, nbytes.value, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert torch.equal(out, w8a8_block_fp8_matmul(a, b, sa, sb, [128, 128], torch.float32))
    assert bool((ws[n:] == 123.0).all())
    used = int((ws[:n] != 123.0).sum())
    assert (used > 0) == (split.value > 1)
