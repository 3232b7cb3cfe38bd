"""The work a server has the block-FP8 path do, as timed cases.

Every case goes through the entry points that a model's layers call, on the layer sizes of the repository's
benchmark configurations (dense MLP, attention projections, expert layer) at decode and prefill token counts:

  linear      Fp8LinearMethod.apply: quantise the activations, multiply with the block-quantised weight, add the bias
  mlp         gate_up projection -> SiLU * mul -> down projection
  moe         routing, then the fused expert layer
  quant       the activation quantiser alone, for callers that feed their own product
  norm_quant  residual add + RMSNorm + quantisation, the producer of a linear's input

`scales` is "fp32" (amax / 448 scales) or "ue8m0" (power-of-two scales, the mode that the weights are re-quantised
for at load time).  Weights and activations are synthetic: N(0, 0.02) and N(0, 1).
"""
import torch

from sglang_b200 import sgl_kernel
from sglang_b200.layers.moe.cutlass_moe import fused_experts_block_fp8_ue8m0
from sglang_b200.layers.moe.topk import fused_topk
from sglang_b200.layers.quantization.deep_gemm_wrapper import gate_up_silu_quant_pow2
from sglang_b200.layers.quantization.fp8 import Fp8Config, Fp8LinearMethod, Fp8MoEMethod
from sglang_b200.layers.quantization.fp8_kernel import (rmsnorm_per_token_group_quant_fp8,
                                                        sglang_per_token_group_quant_fp8,
                                                        w8a8_block_fp8_matmul_deepgemm)
from sglang_b200.layers.quantization.fp8_utils import ceil_to_ue8m0

BLOCK = [128, 128]
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}

# (K, N) of the projections in the benchmark configurations, with the shards that 2, 4 and 8 ranks hold
PROJECTIONS = [
    (7168, 36864), (18432, 7168), (7168, 4096), (7168, 576),                      # gate_up, down, config 0, kv_a (ragged)
    (8192, 10240), (8192, 57344), (8192, 8192), (28672, 8192),                    # qkv, gate_up, o, down
    (8192, 5120), (8192, 1280), (8192, 7168), (4096, 8192), (1024, 8192), (3584, 8192), (14336, 8192),
    (7168, 4608), (2304, 7168), (9216, 7168),
]
# (hidden, intermediate) of the dense MLPs, whole and sharded
MLPS = [(7168, 18432), (7168, 4608), (7168, 2304), (8192, 28672), (8192, 7168), (8192, 3584)]
# (experts, hidden, intermediate, top-k): the 256-expert layer, an eighth of it, and layers of fewer or smaller experts
EXPERT_LAYERS = [(256, 7168, 2048, 8), (32, 7168, 2048, 8), (64, 2048, 1408, 6), (128, 4096, 1536, 8), (8, 4096, 2048, 2)]


def listed():
    return [
        # one request decoding: the latency of a single small call, launches and host work included
        {"name": "linear_1_o_proj", "kind": "linear", "scales": "fp32", "dtype": "bf16", "bias": False,
         "M": 1, "K": 8192, "N": 8192},
        # a small decode batch on a long-K projection, power-of-two scales
        {"name": "linear_ue8m0_16_down", "kind": "linear", "scales": "ue8m0", "dtype": "bf16", "bias": False,
         "M": 16, "K": 18432, "N": 7168},
        # benchmark configuration 0: a decode batch of 64
        {"name": "linear_64_config0", "kind": "linear", "scales": "fp32", "dtype": "bf16", "bias": False,
         "M": 64, "K": 7168, "N": 4096},
        # a large decode batch through an fp16 qkv projection with bias
        {"name": "linear_128_qkv_bias", "kind": "linear", "scales": "fp32", "dtype": "fp16", "bias": True,
         "M": 128, "K": 8192, "N": 10240},
        # a chunk of prefill with an odd token count through the ragged kv_a projection (N = 576)
        {"name": "linear_1021_kv_a", "kind": "linear", "scales": "fp32", "dtype": "bf16", "bias": False,
         "M": 1021, "K": 7168, "N": 576},
        # prefill through the dense MLP: the benchmark's headline step
        {"name": "mlp_4096", "kind": "mlp", "scales": "fp32", "dtype": "bf16", "M": 4096, "K": 7168, "I": 18432},
        # a long prefill through the same MLP with power-of-two scales
        {"name": "mlp_ue8m0_8192", "kind": "mlp", "scales": "ue8m0", "dtype": "bf16", "M": 8192, "K": 7168, "I": 18432},
        # a decode batch through the 256-expert layer: nearly every routed row is an expert of its own
        {"name": "moe_16_e256", "kind": "moe", "scales": "fp32", "dtype": "bf16", "M": 16, "E": 256, "H": 7168,
         "I": 2048, "topk": 8},
        # prefill through the 256-expert layer: 128 rows an expert
        {"name": "moe_4096_e256", "kind": "moe", "scales": "fp32", "dtype": "bf16", "M": 4096, "E": 256, "H": 7168,
         "I": 2048, "topk": 8},
        # the share of one expert-parallel rank, power-of-two scales, an odd token count
        {"name": "moe_ue8m0_515_e32", "kind": "moe", "scales": "ue8m0", "dtype": "bf16", "M": 515, "E": 32, "H": 7168,
         "I": 2048, "topk": 8},
        # benchmark configuration 2: the quantiser alone, column-major scales, activations with outliers
        {"name": "quant_16384", "kind": "quant", "scales": "fp32", "dtype": "bf16", "column_major": True,
         "M": 16384, "K": 7168},
        # what precedes a projection in every layer: residual add, RMSNorm, quantisation
        {"name": "norm_quant_2048", "kind": "norm_quant", "scales": "fp32", "dtype": "bf16", "M": 2048, "K": 7168},
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["mlp"] * 2 + ["moe"] * 3 + ["quant", "norm_quant"])
    scales = rng.choice(["fp32", "fp32", "ue8m0"])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "linear":
        K, N = rng.choice(PROJECTIONS)
        most = min(16384, int(3.0e12 / (2.0 * K * N)))
        if scales == "ue8m0":
            dtype = "bf16"      # the power-of-two mode takes bf16 activations and whole 128-wide weight blocks
            N = (N + 127) // 128 * 128
        return {"kind": kind, "scales": scales, "dtype": dtype, "bias": rng.random() < 0.25,
                "M": _log_uniform(rng, 1, most), "K": K, "N": N}
    if kind == "mlp":
        K, I = rng.choice(MLPS)
        most = min(16384, int(3.0e12 / (6.0 * K * I)))
        return {"kind": kind, "scales": scales, "dtype": "bf16" if scales == "ue8m0" else dtype,
                "M": _log_uniform(rng, 1, most), "K": K, "I": I}
    if kind == "moe":
        E, H, I, topk = rng.choice(EXPERT_LAYERS)
        return {"kind": kind, "scales": scales, "dtype": dtype, "M": _log_uniform(rng, 1, 4096), "E": E, "H": H, "I": I,
                "topk": topk}
    K = 128 * _log_uniform(rng, 8, 128)
    M = _log_uniform(rng, 1, 16384)
    if kind == "quant":
        return {"kind": kind, "scales": scales, "dtype": dtype, "column_major": rng.random() < 0.5, "M": M, "K": K}
    return {"kind": kind, "scales": scales, "dtype": dtype, "M": M, "K": K}


# ------------------------------------------------------------------------------------------------ inputs
def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)


def _block_weight_into(gen, codes, scale, pow2):
    """codes [N, K] e4m3 and scale [ceil(N/128), ceil(K/128)] <- an N(0, 0.02) weight quantised per 128 x 128 block."""
    N, K = codes.shape
    step = 4096
    for n0 in range(0, N, step):
        n1 = min(N, n0 + step)
        rows, nb, kb = n1 - n0, (n1 - n0 + 127) // 128, (K + 127) // 128
        w = _randn(gen, rows, K).mul_(0.02)
        if rows % 128 or K % 128:
            w = torch.nn.functional.pad(w, (0, kb * 128 - K, 0, nb * 128 - rows))
        w = w.view(nb, 128, kb, 128)
        s = w.abs().amax(dim=(1, 3), keepdim=True).clamp_(min=1e-4).div_(448.0)
        if pow2:
            s = ceil_to_ue8m0(s)
        codes[n0:n1] = w.div_(s).view(nb * 128, kb * 128)[:rows, :K].to(torch.float8_e4m3fn)
        scale[n0 // 128: n0 // 128 + nb] = s.view(nb, kb)


def _activations(gen, M, K, dtype):
    return _randn(gen, M, K).to(dtype)


def _linear_layer(gen, N, K, dtype, ue8m0):
    method = Fp8LinearMethod(Fp8Config(is_checkpoint_fp8_serialized=True, activation_scheme="dynamic",
                                       weight_block_size=BLOCK), scale_ue8m0=ue8m0)
    layer = torch.nn.Module()
    method.create_weights(layer, K, [N], K, N, dtype, device=torch.device("cuda"))
    _block_weight_into(gen, layer.weight.data, layer.weight_scale_inv.data, False)
    method.process_weights_after_loading(layer)
    return method, layer


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype, ue8m0 = DTYPES[case["dtype"]], case["scales"] == "ue8m0"
    kind, M = case["kind"], case["M"]
    state = {"case": case}
    if kind == "linear":
        K, N = case["K"], case["N"]
        state["method"], state["layer"] = _linear_layer(gen, N, K, dtype, ue8m0)
        state["bias"] = _randn(gen, N).to(dtype) if case["bias"] else None
        state["x"] = _activations(gen, M, K, dtype)
    elif kind == "mlp":
        K, I = case["K"], case["I"]
        state["method"], state["gate_up"] = _linear_layer(gen, 2 * I, K, dtype, ue8m0)
        _, state["down"] = _linear_layer(gen, K, I, dtype, ue8m0)
        state["x"] = _activations(gen, M, K, dtype)
    elif kind == "moe":
        E, H, I = case["E"], case["H"], case["I"]
        method = Fp8MoEMethod(Fp8Config(is_checkpoint_fp8_serialized=True, activation_scheme="dynamic",
                                        weight_block_size=BLOCK))
        layer = torch.nn.Module()
        method.create_weights(layer, E, H, I, dtype, device=torch.device("cuda"))
        _block_weight_into(gen, layer.w13_weight.data.view(E * 2 * I, H),
                           layer.w13_weight_scale_inv.data.view(E * 2 * I // 128, H // 128), ue8m0)
        _block_weight_into(gen, layer.w2_weight.data.view(E * H, I),
                           layer.w2_weight_scale_inv.data.view(E * H // 128, I // 128), ue8m0)
        method.process_weights_after_loading(layer)
        state["method"], state["layer"] = method, layer
        state["x"] = _activations(gen, M, H, dtype)
        state["logits"] = _randn(gen, M, E)
        state["choice_bias"] = _randn(gen, E).mul_(0.1)
    elif kind == "quant":
        K = case["K"]
        x = _randn(gen, M, K)
        x[torch.rand(M, K, generator=gen, device="cuda") < 1e-3] *= 100.0
        state["x"] = x.to(dtype)
    else:
        K = case["K"]
        state["x"] = _activations(gen, M, K, dtype)
        state["residual"] = _activations(gen, M, K, dtype)
        state["weight"] = (1.0 + 0.1 * _randn(gen, K)).to(dtype)
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _run_mlp(state):
    if state["case"]["scales"] == "fp32":
        h = state["method"].apply(state["gate_up"], state["x"])
        return state["method"].apply(state["down"], sgl_kernel.silu_and_mul(h))
    gate_up, down = state["gate_up"], state["down"]
    q, s = sglang_per_token_group_quant_fp8(state["x"], 128, column_major_scales=True, scale_tma_aligned=True,
                                            scale_ue8m0=True)
    q2, s2 = gate_up_silu_quant_pow2(q, s, gate_up.weight.data, gate_up.weight_scale_inv.data)
    return w8a8_block_fp8_matmul_deepgemm(q2, down.weight.data, s2, down.weight_scale_inv.data, BLOCK, torch.bfloat16,
                                          weight_scale_ue8m0=True)


def _run_moe(state):
    case, layer, x = state["case"], state["layer"], state["x"]
    if case["E"] == 256:        # grouped sigmoid gate: 8 groups, the best 4 stay
        topk = sgl_kernel.moe_fused_gate(state["logits"], state["choice_bias"], 8, 4, case["topk"])
    else:                       # softmax router
        topk = fused_topk(x, state["logits"], case["topk"], True)
    if case["scales"] == "fp32":
        return state["method"].apply(layer, x, topk)
    return fused_experts_block_fp8_ue8m0(x, layer.w13_weight.data, layer.w2_weight.data, layer.w13_weight_scale_inv.data,
                                         layer.w2_weight_scale_inv.data, topk[0], topk[1])


def run(state):
    case = state["case"]
    kind, ue8m0 = case["kind"], case["scales"] == "ue8m0"
    if kind == "linear":
        return state["method"].apply(state["layer"], state["x"], state["bias"])
    if kind == "mlp":
        return _run_mlp(state)
    if kind == "moe":
        return _run_moe(state)
    if kind == "quant":
        column_major = case["column_major"] or ue8m0
        return sglang_per_token_group_quant_fp8(state["x"], 128, column_major_scales=column_major,
                                                scale_tma_aligned=column_major, scale_ue8m0=ue8m0)
    # the residual stream is updated in place, as between the layers of a model
    q, s = rmsnorm_per_token_group_quant_fp8(state["x"], state["weight"], 1e-6, state["residual"],
                                             column_major_scales=True, scale_tma_aligned=True, scale_ue8m0=ue8m0)
    return q, s, state["residual"]


# ------------------------------------------------------------------------------------------------ what a pass needs
def _weight_bytes(N, K):
    return N * K + 4 * ((N + 127) // 128) * ((K + 127) // 128)


def work(case):
    kind, M, ue8m0 = case["kind"], case["M"], case["scales"] == "ue8m0"
    if kind == "linear":
        K, N = case["K"], case["N"]
        return {"bytes": 2 * M * (K + N) + _weight_bytes(N, K) + (2 * N if case["bias"] else 0), "flops": 2.0 * M * N * K}
    if kind == "mlp":
        K, I = case["K"], case["I"]
        return {"bytes": 4 * M * K + _weight_bytes(2 * I, K) + _weight_bytes(K, I), "flops": 6.0 * M * K * I}
    if kind == "moe":
        E, H, I, topk = case["E"], case["H"], case["I"], case["topk"]
        touched = E * (1.0 - (1.0 - topk / E) ** M)       # experts that get a row, in the mean
        return {"bytes": 4 * M * H + 4 * M * E + touched * (_weight_bytes(2 * I, H) + _weight_bytes(H, I)),
                "flops": 6.0 * M * topk * H * I}
    K = case["K"]
    scale_bytes = M * ((K + 511) // 512) * 4 if ue8m0 else M * (K // 128) * 4
    if kind == "quant":
        return {"bytes": 3 * M * K + scale_bytes, "flops": 4.0 * M * K}
    # x and the residual read, the residual and the codes written
    return {"bytes": 7 * M * K + scale_bytes, "flops": 8.0 * M * K}


def tolerance(case):
    if case["kind"] == "quant":
        return "exact"          # codes and scales are fixed bit for bit
    if case["kind"] == "norm_quant":
        # the order of the sum of squares can move a value to the neighbouring 16-bit number, and with it a code by one
        # step (1/8 of the value) or a power-of-two scale by one
        return {"rel": 2e-3, "max": 0.2, "differ": 1e-3}
    if case["kind"] == "linear":
        return {"rel": 3e-3, "max": 0.05}      # one rounding to a 16-bit result after fp32 sums in another order
    # two products with an 8-bit quantisation between them: a sum in another order moves a few codes by one step
    return {"rel": 1e-2, "max": 0.2}
