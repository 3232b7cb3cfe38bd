"""GPU: the linear at decode sizes (quantiser, product, split sum and bias as one chain) against the oracle's two steps."""
import pytest
import torch

from oracle import block_fp8_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 17, 33, 64, 65, 192])
@pytest.mark.parametrize("N,K", [(128, 128), (576, 7168), (1280, 1152), (19200, 384)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_decode_linear_matches_the_oracle(M, N, K, dtype):
    from sglang_b200.layers.quantization.fp8_utils import w8a8_block_fp8_linear
    g = torch.Generator().manual_seed(M * 31 + N + K)
    x = torch.randn(M, K, generator=g).to(dtype)
    x[0, :128] = 0                                              # an all-zero group
    wq, ws = O.gen_weight((N + 127) // 128 * 128, K, seed=N + K)
    wq = wq[:N].contiguous()
    bias = torch.randn(N, generator=g).to(dtype)
    q, s = O.quant_group_fp8_cuda_semantics(x, 128)
    ref = O.block_fp8_matmul_fp32(q, wq, s, ws).to(dtype)
    xd, wd, wsd = x.cuda(), wq.cuda(), ws.cuda()
    for _ in range(2):
        out = w8a8_block_fp8_linear(xd, wd, [128, 128], wsd)
    assert O.rel_l2(out.cpu().float(), ref.float()) <= 1e-3
    with_bias = w8a8_block_fp8_linear(xd, wd, [128, 128], wsd, bias=bias.cuda())
    out += bias.cuda()
    assert torch.equal(out, with_bias)


@pytest.mark.parametrize("M,N", [(1, 640), (31, 640), (64, 640), (65, 9600), (192, 9600), (193, 640), (512, 1280),
                                 (513, 1280), (1023, 8192), (1024, 640)])
def test_decode_linear_power_of_two_scales(M, N):
    from sglang_b200.layers.quantization.fp8_kernel import sglang_per_token_group_quant_fp8, w8a8_block_fp8_matmul_deepgemm
    from sglang_b200.layers.quantization.fp8_utils import (deepgemm_w8a8_block_fp8_linear_with_fallback,
                                                            requant_weight_ue8m0)
    K = 2304
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=g, device="cuda").to(torch.bfloat16)
    wq, ws = O.gen_weight(N, K, seed=9)
    wq, ws = requant_weight_ue8m0(wq.cuda(), ws.cuda(), [128, 128])
    out = deepgemm_w8a8_block_fp8_linear_with_fallback(x, wq, [128, 128], ws, weight_scale_ue8m0=True)
    q, s = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
    ref = w8a8_block_fp8_matmul_deepgemm(q, wq, s, ws, [128, 128], torch.bfloat16, weight_scale_ue8m0=True)
    assert O.rel_l2(out.float().cpu(), ref.float().cpu()) <= 1e-3
    q_f, s_f, w_f = q.float().view(M, -1, 128), s, wq.float().view(N // 128, 128, K // 128, 128)
    byte = torch.stack([(s_f >> (8 * b)) & 0xff for b in range(4)], dim=-1).reshape(M, -1)[:, :K // 128]
    a_f = (q_f * torch.exp2(byte.float() - 127).unsqueeze(-1)).view(M, K)
    b_f = (w_f * ws.view(N // 128, 1, K // 128, 1)).reshape(N, K)
    exact = (a_f.double() @ b_f.double().T).to(torch.bfloat16)
    assert O.rel_l2(ref.float().cpu(), exact.float().cpu()) <= 1e-3


@pytest.mark.parametrize("pow2_weights", [False, True])
@pytest.mark.parametrize("M,N,K", [(16, 1280, 8192), (200, 640, 7168)])
def test_power_of_two_linear_obeys_the_split_switch(M, N, K, pow2_weights, monkeypatch):
    """Sizes that the automatic mode splits: with the switch off, the bits of the unsplit product."""
    from sglang_b200.layers.quantization.fp8_kernel import sglang_per_token_group_quant_fp8, w8a8_block_fp8_matmul_deepgemm
    from sglang_b200.layers.quantization.fp8_utils import (deepgemm_w8a8_block_fp8_linear_with_fallback,
                                                            requant_weight_ue8m0)
    from sglang_b200.sgl_kernel import gemm
    x = torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    wq, ws = O.gen_weight(N, K, seed=N)
    wq, ws = requant_weight_ue8m0(wq.cuda(), ws.cuda(), [128, 128])
    q, s = sglang_per_token_group_quant_fp8(x, 128, column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=True)
    unsplit = w8a8_block_fp8_matmul_deepgemm(q, wq, s, ws, [128, 128], torch.bfloat16, weight_scale_ue8m0=pow2_weights)
    assert gemm._splitk_plan(M, N, K, x.device)[0] > 1, "the sizes are meant to be split"
    monkeypatch.setattr(gemm, "SPLIT_K_MODE", "off")
    out = deepgemm_w8a8_block_fp8_linear_with_fallback(x, wq, [128, 128], ws, weight_scale_ue8m0=pow2_weights)
    assert torch.equal(out, unsplit)
