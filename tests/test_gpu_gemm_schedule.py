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
