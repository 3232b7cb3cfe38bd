"""GPU: the expert layer's one-call chain (routing tables in one launch, tokens quantised straight to their experts' rows,
column-split weighted sum) around the sizes where its kernels change: 4096 routed ids, a K that is no multiple of 512."""
import pytest
import torch

from oracle import block_fp8_oracle as O

pytestmark = pytest.mark.gpu


def _case(m, topk, E, n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randn(m, k, generator=g, device="cuda").to(dtype)
    w13, s13 = O.gen_weight(E * 2 * n, k, seed=1)
    w2, s2 = O.gen_weight(E * k, n, seed=2)
    ids = torch.rand(m, E, generator=g, device="cuda").topk(topk, dim=-1).indices.to(torch.int32)
    ids[:, 0] = torch.where(torch.arange(m, device="cuda") % 3 == 0, -1, ids[:, 0])      # masked choices
    w = torch.rand(m, topk, generator=g, device="cuda")
    return (x, w13.view(E, 2 * n, k).cuda(), w2.view(E, k, n).cuda(), s13.view(E, 2 * n // 128, k // 128).cuda(),
            s2.view(E, k // 128, n // 128).cuda(), w, ids)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,topk,E,k", [(1, 8, 9, 128), (33, 3, 40, 640), (512, 8, 16, 384), (513, 8, 16, 2304)])
def test_expert_chain_equals_its_stages(m, topk, E, k, dtype):
    from sglang_b200.layers.moe.cutlass_moe import fused_experts_block_fp8, fused_experts_block_fp8_ue8m0
    from sglang_b200.layers.quantization.fp8_utils import requant_weight_ue8m0
    n = 256
    x, w13, w2, s13, s2, w, ids = _case(m, topk, E, n, k, dtype)
    out = fused_experts_block_fp8(x, w13, w2, s13, s2, w, ids)
    ref = O.cutlass_fused_experts_fp8(x.cpu(), w13.cpu(), w2.cpu(), s13.cpu(), s2.cpu(),
                                      torch.where(ids < 0, 0, w).cpu(), ids.clamp(min=0).cpu())
    assert O.rel_l2(out.float().cpu(), ref.float()) <= 5e-3
    parts = [[requant_weight_ue8m0(a, b, [128, 128]) for a, b in zip(q, s)] for q, s in ((w13, s13), (w2, s2))]
    (w13p, s13p), (w2p, s2p) = [(torch.stack([p[0] for p in l]), torch.stack([p[1] for p in l])) for l in parts]
    args = (x, w13p, w2p, s13p, s2p, w, ids)
    assert torch.equal(fused_experts_block_fp8_ue8m0(*args), fused_experts_block_fp8_ue8m0(*args, fuse_activation=False))
