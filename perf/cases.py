"""Performance cases of the MoE block: what a user's program has it do, through its public entry points.

Two models run on the block: one whose experts are bf16, and one whose experts are GPTQ int4 (W4A16).  A
serving program prefills prompts with them (hundreds to thousands of tokens a call, the lengths as the prompts
come) and decodes small batches (one token per sequence).  It calls the block eagerly, or captures it, or a
chain of decoder layers' MoE halves, into a CUDA graph.  Beside the block stand the single W4A16 linear (the
attention projections of the quantised model), the separate kernel functions that the reference's own layer is
written with, and small fp32 layers.

Sizes are those of the repository's configurations and tests: the Qwen3-30B-A3B layer (hidden 2048, 128
experts, 8 per token, expert width 768), smaller layers with it, and batches of 1 to 16384 tokens.
"""
import os
import sys

import torch
import torch.nn.functional as F

sys.path.insert(1, os.path.join(os.getcwd(), "mini-qwen-llm_b200"))

from mini_qwen_b200 import Qwen3MoEConfig, synthetic  # noqa: E402
from mini_qwen_b200.graph import CapturedForward  # noqa: E402
from mini_qwen_b200.kernels import moe_grouped_gemm, moe_permute, moe_router, moe_unpermute  # noqa: E402
from mini_qwen_b200.model.layers import LinearW4A16, Qwen3MoEBlock, RMSNorm  # noqa: E402

GROUP = 128
QWEN = {"H": 2048, "E": 128, "K": 8, "I": 768}


def listed():
    return [
        # one sequence being decoded on the quantised model, the block called eagerly: the smallest call
        {"name": "w4_decode_1", "kind": "w4", "T": 1, "graph": False, "half": False, **QWEN},
        # a batch of 64 sequences, the layer replayed from its CUDA graph
        {"name": "w4_decode_64_graph", "kind": "w4", "T": 64, "graph": True, "half": False, **QWEN},
        # 16 sequences through the MoE halves (norm, block, residual) of 16 decoder layers in one graph
        {"name": "w4_stack_16", "kind": "w4_stack", "T": 16, "layers": 16, **QWEN},
        # a prompt of 512 tokens on the quantised model, as a decoder layer's half
        {"name": "w4_prefill_512", "kind": "w4", "T": 512, "graph": False, "half": True, **QWEN},
        # a long prompt, or several together
        {"name": "w4_prefill_4096", "kind": "w4", "T": 4096, "graph": False, "half": False, **QWEN},
        # attention projections of the quantised model: one token, and a prompt of odd length
        {"name": "w4_linear_1", "kind": "w4_linear", "M": 1, "Kd": 2048, "N": 4096},
        {"name": "w4_linear_500", "kind": "w4_linear", "M": 500, "Kd": 4096, "N": 2048},
        # eight sequences being decoded on the bf16 model, as a decoder layer's half
        {"name": "bf16_decode_8", "kind": "bf16", "T": 8, "half": True, "skew": 0.0, **QWEN},
        # the kernel functions one by one, as the reference's layer calls them; prompts of odd length
        {"name": "bf16_functions_777", "kind": "functions", "T": 777, **QWEN},
        # bf16 prefill of 4096 tokens
        {"name": "bf16_prefill_4096", "kind": "bf16", "T": 4096, "half": False, "skew": 0.0, **QWEN},
        # 16384 tokens whose experts' popularity follows Zipf's law: thousands of rows for some, none for others
        {"name": "bf16_skewed_16384", "kind": "bf16", "T": 16384, "half": False, "skew": 1.2, **QWEN},
        # a small fp32 layer
        {"name": "fp32_small_64", "kind": "fp32", "T": 64, "H": 256, "E": 8, "K": 2, "I": 512},
    ]


def _log_int(rng, lo, hi):
    """A whole number of lo..hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _layer_shape(rng):
    """The Qwen3-30B-A3B layer, or one no larger of the same family."""
    if rng.random() < 0.6:
        return dict(QWEN)
    E = rng.choice([16, 32, 64, 128])
    return {"H": 256 * rng.randint(2, 8), "E": E, "K": rng.choice([2, 4, 6, 8]), "I": 128 * rng.randint(2, 6)}


def draw(rng):
    kind = rng.choice(["w4_decode", "w4_decode", "w4_stack", "w4_prefill", "w4_prefill", "w4_linear", "w4_linear",
                       "bf16_decode", "bf16_prefill", "bf16_prefill", "functions", "fp32"])
    if kind == "w4_decode":
        return {"kind": "w4", "T": _log_int(rng, 1, 64), "graph": rng.random() < 0.5, "half": rng.random() < 0.5,
                **_layer_shape(rng)}
    if kind == "w4_stack":
        return {"kind": "w4_stack", "T": _log_int(rng, 1, 64), "layers": rng.randint(4, 16), **_layer_shape(rng)}
    if kind == "w4_prefill":
        return {"kind": "w4", "T": _log_int(rng, 65, 4096), "graph": False, "half": rng.random() < 0.5,
                **_layer_shape(rng)}
    if kind == "w4_linear":
        return {"kind": "w4_linear", "M": _log_int(rng, 1, 2048), "Kd": 128 * rng.randint(4, 32),
                "N": 64 * rng.randint(8, 64)}
    if kind == "bf16_decode":
        return {"kind": "bf16", "T": _log_int(rng, 1, 64), "half": rng.random() < 0.5, "skew": 0.0,
                **_layer_shape(rng)}
    if kind == "bf16_prefill":
        return {"kind": "bf16", "T": _log_int(rng, 65, 16384), "half": rng.random() < 0.5,
                "skew": rng.choice([0.0, 0.0, 1.2]), **_layer_shape(rng)}
    if kind == "functions":
        return {"kind": "functions", "T": _log_int(rng, 16, 4096), **_layer_shape(rng)}
    return {"kind": "fp32", "T": _log_int(rng, 1, 256), "H": 64 * rng.randint(2, 8), "E": rng.choice([8, 16, 32]),
            "K": rng.choice([2, 4]), "I": 64 * rng.randint(2, 8)}


# ---- inputs ---------------------------------------------------------------------------------------------
def _normal(gen, shape, std, dtype):
    return torch.empty(shape, dtype=dtype, device=gen.device).normal_(0.0, std, generator=gen)


def _bits(gen, shape):
    return torch.randint(-2 ** 31, 2 ** 31 - 1, shape, generator=gen, device=gen.device, dtype=torch.int32)


def _w4(gen, lead, kd, n):
    """Packed int4 weights as a quantised checkpoint holds them: bell-shaped around the zero point (the sum of
    two uniform 0..7 and one bit), zero points 7 or 8, scales such that a weight is about N(0, 0.02)."""
    qw = (_bits(gen, (*lead, kd // 8, n)) & 0x77777777) + (_bits(gen, (*lead, kd // 8, n)) & 0x77777777)
    qw = qw + (_bits(gen, (*lead, kd // 8, n)) & 0x11111111)
    scales = (torch.rand(*lead, kd // GROUP, n, generator=gen, device=gen.device) * 0.003 + 0.0045).to(torch.bfloat16)
    qz = (_bits(gen, (*lead, kd // GROUP, n // 8)) & 0x11111111) + 0x77777777
    return qw, scales, qz


def _w4_block(gen, c):
    H, E, I = c["H"], c["E"], c["I"]
    cfg = Qwen3MoEConfig(hidden_size=H, intermediate_size=I, num_experts=E, num_experts_per_tok=c["K"])
    router = _normal(gen, (E, H), 0.02, torch.bfloat16)
    return Qwen3MoEBlock.from_stacked_w4(cfg, router, _w4(gen, (E,), H, I), _w4(gen, (E,), H, I), _w4(gen, (E,), I, H),
                                         GROUP)


def _dense_block(gen, c, dtype):
    H, E, I = c["H"], c["E"], c["I"]
    cfg = Qwen3MoEConfig(hidden_size=H, intermediate_size=I, num_experts=E, num_experts_per_tok=c["K"])
    router = _normal(gen, (E, H), 0.02, dtype)
    return Qwen3MoEBlock.from_stacked(cfg, router, _normal(gen, (E, 2 * I, H), 0.02, dtype),
                                      _normal(gen, (E, H, I), 0.02, dtype))


def _norm(gen, H, dtype):
    norm = RMSNorm(H)
    norm.weight = torch.nn.Parameter(1.0 + _normal(gen, (H,), 0.1, dtype), requires_grad=False)
    return norm


def _call(block, norm):
    """The call of a layer: the block alone, or norm, block and residual."""
    return block if norm is None else (lambda h: block.half_layer(h, norm))


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = c["kind"]
    if kind == "w4_linear":
        lin = LinearW4A16(c["Kd"], c["N"], GROUP)
        lin.qweight, lin.scales, lin.qzeros = _w4(gen, (), c["Kd"], c["N"])
        return {"kind": kind, "layer": lin, "x": _normal(gen, (c["M"], c["Kd"]), 1.0, torch.bfloat16)}
    dtype = torch.float32 if kind == "fp32" else torch.bfloat16
    x = _normal(gen, (c["T"], c["H"]), 1.0, dtype)
    if kind == "functions":
        H, E, I = c["H"], c["E"], c["I"]
        return {"kind": kind, "x": x, "top_k": c["K"], "router": _normal(gen, (E, H), 0.02, dtype),
                "gate": _normal(gen, (E, I, H), 0.02, dtype), "up": _normal(gen, (E, I, H), 0.02, dtype),
                "down": _normal(gen, (E, H, I), 0.02, dtype)}
    if kind == "w4_stack":
        layers = [(_w4_block(gen, c), _norm(gen, c["H"], dtype)) for _ in range(c["layers"])]

        def stack(h):
            for block, norm in layers:
                h = block.half_layer(h, norm)
            return h

        return {"kind": "graph", "graph": CapturedForward(stack, x), "x": x, "keep": layers}
    if kind == "w4":
        block = _w4_block(gen, c)
    else:
        block = _dense_block(gen, c, dtype)
        if c.get("skew"):
            block.router_bias = synthetic.zipf_router_bias(seed, c["E"], s=c["skew"]).cuda()
    layer = _call(block, _norm(gen, c["H"], dtype) if c.get("half") else None)
    if c.get("graph"):
        return {"kind": "graph", "graph": CapturedForward(layer, x), "x": x, "keep": layer}
    return {"kind": "layer", "layer": layer, "x": x}


@torch.no_grad()
def run(state):
    kind, x = state["kind"], state["x"]
    if kind == "graph":
        state["graph"].x.copy_(x)
        return state["graph"].replay()
    if kind != "functions":
        return state["layer"](x)
    # the reference's layer, function by function
    ids, weights = moe_router(x, state["router"], state["top_k"])
    weights = weights / weights.sum(dim=-1, keepdim=True)
    rows, offsets = moe_permute(x, ids, state["router"].shape[0])
    h = F.silu(moe_grouped_gemm(rows, state["gate"], offsets)) * moe_grouped_gemm(rows, state["up"], offsets)
    y = moe_grouped_gemm(h, state["down"], offsets)
    return {"ids": ids, "weights": weights, "offsets": offsets, "out": moe_unpermute(y, weights, ids, x.shape[0])}


# ---- what a pass cannot do without ----------------------------------------------------------------------
def _w4_bytes(kd, n):
    return kd * n // 2 + (kd // GROUP) * n * 2 + (kd // GROUP) * n // 2


def _experts_hit(c):
    """Experts that at least one of the tokens chose, in the mean over evenly popular experts; every expert's
    popularity under Zipf's law is (rank ** -s) in odds."""
    E, K, T = c["E"], c["K"], c["T"]
    p = [(r + 1) ** -c.get("skew", 0.0) for r in range(E)]
    total = sum(p)
    return sum(1.0 - (1.0 - min(1.0, K * v / total)) ** T for v in p)


def work(case):
    c = case
    if c["kind"] == "w4_linear":
        M, Kd, N = c["M"], c["Kd"], c["N"]
        return {"bytes": _w4_bytes(Kd, N) + 2 * M * (Kd + N), "flops": 2 * M * Kd * N}
    H, E, K, I, T = c["H"], c["E"], c["K"], c["I"], c["T"]
    size = 4 if c["kind"] == "fp32" else 2
    if c["kind"].startswith("w4"):
        expert = 2 * _w4_bytes(H, I) + _w4_bytes(I, H)
    else:
        expert = 3 * H * I * size
    layers = c.get("layers", 1)
    per_layer = _experts_hit(c) * expert + E * H * size
    nbytes = layers * per_layer + 2 * T * H * size
    if c["kind"] == "functions":     # the functions hand rows over in memory: each reads its inputs and writes its result
        S = T * K
        nbytes += size * (2 * T * H + 3 * S * H + 3 * S * I + S * H + S * I) + 2 * S * 12
    return {"bytes": nbytes, "flops": layers * (2 * T * K * 3 * H * I + 2 * T * H * E)}


def tolerance(case):
    """fp32 layers: sums of a few hundred fp32 products in another order.  The others: bf16 roundings between the
    operations of an expert; a routing id may differ where two experts' scores tie in fp32."""
    if case["kind"] == "fp32":
        return {"rel": 1e-5}
    if case["kind"] == "functions":
        return {"rel": 1e-2, "differ": 1e-3}
    return {"rel": 1e-2}
