"""The whole-block call (csrc/block.cu) against the same chain issued stage by stage: the same kernels on the same
inputs, so identical bits, in every branch of its dispatch (decode and prefill batches on both sides of the 64-token
line, dense layers with and without the tcgen05 kernels, W4A16 layers on the stream, tile and fallback kernels, norm
and residual)."""
import copy
import pickle

import pytest
import torch

from mini_qwen_b200 import Qwen3MoEConfig, synthetic
from mini_qwen_b200.model.layers import Qwen3MoEBlock, RMSNorm

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def make(kind, E, K, H, I, group=128):
    g = torch.Generator(device=DEV).manual_seed(E + H)
    cfg = Qwen3MoEConfig(hidden_size=H, intermediate_size=I, num_experts=E, num_experts_per_tok=K)
    dt = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "w4": torch.bfloat16}[kind]
    router = (torch.randn(E, H, generator=g, device=DEV) * 0.05).to(dt)
    if kind == "w4":
        return Qwen3MoEBlock.from_stacked_w4(cfg, router, *synthetic.w4a16_stacks_on_device(DEV, 7, E, H, I, group), group), dt
    rnd = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.02).to(dt)
    return Qwen3MoEBlock.from_stacked(cfg, router, rnd(E, 2 * I, H), rnd(E, H, I)), dt


@pytest.mark.parametrize("kind,E,K,H,I,group", [
    ("bf16", 16, 4, 256, 128, 0), ("bf16", 8, 2, 96, 40, 0), ("fp16", 8, 2, 128, 128, 0), ("fp32", 8, 2, 64, 32, 0),
    ("w4", 16, 4, 256, 128, 128), ("w4", 32, 8, 128, 256, 128), ("w4", 8, 2, 128, 64, 32)])
@pytest.mark.parametrize("T", [1, 17, 64, 65, 200])
def test_whole_block_call_equals_the_staged_chain(kind, E, K, H, I, group, T):
    blk, dt = make(kind, E, K, H, I, group)
    g = torch.Generator(device=DEV).manual_seed(T)
    x = torch.randn(T, H, generator=g, device=DEV).to(dt)
    res = torch.randn(T, H, generator=g, device=DEV).to(dt)
    norm = RMSNorm(H)
    norm.weight = torch.nn.Parameter(1 + 0.1 * torch.randn(H, generator=g, device=DEV).to(dt), requires_grad=False)
    for bias in (None, torch.linspace(-1, 1, E, device=DEV)):
        blk.router_bias = bias
        assert blk._native_layer() is not None
        got = blk(x), blk(x, residual=res), blk.half_layer(x, norm)
        want = blk._forward_staged(x), blk._forward_staged(x, res), blk._forward_staged(norm(x), x)
        for a, b in zip(got, want):
            assert a.dtype == dt and a.shape == x.shape and torch.equal(a, b)
    blk.check_status()


def test_description_follows_the_layer():
    """A replaced router, bias or expert weight reaches the next call; copies and pickles make their own description."""
    blk, dt = make("bf16", 8, 2, 128, 128)
    x = torch.randn(9, 128, device=DEV).to(dt)
    blk(x)
    blk.gate.weight = torch.nn.Parameter(-blk.gate.weight.data, requires_grad=False)
    assert torch.equal(blk(x), blk._forward_staged(x))
    rows = blk.gate.weight.data
    blk.gate.weight.data = rows.as_strided((8, 128), (1, 8))        # another layout at the same address
    assert torch.equal(blk(x), blk._forward_staged(x))
    blk.gate.weight.data = rows
    blk.router_bias = torch.linspace(1, -1, 8, device=DEV)
    assert torch.equal(blk(x), blk._forward_staged(x))
    blk.experts[0].gate_proj.weight.data = blk.experts[0].gate_proj.weight.data * 2
    out = blk(x)
    assert torch.equal(out, blk._forward_staged(x))
    for other in (copy.deepcopy(blk), pickle.loads(pickle.dumps(blk))):
        assert torch.equal(other(x), out)
    assert blk(x[:0]).shape == (0, 128)
    with pytest.raises(ValueError):
        blk(x, residual=x[:1])
    with pytest.raises(ValueError):
        blk(x.cpu())


def test_zero_points_off_the_16_byte_grid():
    """Stacks that are views into a flat buffer at a multiple of four bytes: accepted at every batch size, with the
    results of aligned ones (another kernel's order of the fp32 sums, so within a few bf16 roundings)."""
    E, K, H, I = 8, 2, 256, 128
    cfg = Qwen3MoEConfig(hidden_size=H, intermediate_size=I, num_experts=E, num_experts_per_tok=K)
    router = torch.randn(E, H, device=DEV).to(torch.bfloat16)
    stacks = synthetic.w4a16_stacks_on_device(DEV, 7, E, H, I)

    def view(t):
        flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
        flat[1:] = t.reshape(-1)
        return flat[1:].view(t.shape)
    blk = Qwen3MoEBlock.from_stacked_w4(cfg, router, *stacks)
    off = Qwen3MoEBlock.from_stacked_w4(cfg, router, *[(qw, sc, view(qz)) for qw, sc, qz in stacks])
    for T in (3, 64, 65, 400):
        x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
        out = off(x)
        assert torch.equal(out, off._forward_staged(x))
        want = blk(x).float()
        assert float((out.float() - want).norm() / want.norm()) < 1e-2
    off.check_status()
