"""GPU parity of the CTA-pair grouped GEMM (bf16, K % 128 == 0) at the edges of its tile shapes: 128 | 129 and 256 | 257
rows per expert, two tiles of up to 512 rows, tails of one row, one and an odd number of weight sub-tiles."""
import pytest
import torch

from mini_qwen_b200.kernels import moe_grouped_gemm, moe_grouped_swiglu
from mini_qwen_b200.kernels.moe_grouped_gemm import moe_grouped_swiglu_gather
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
# empty groups beside large ones: large averages go to the single-CTA kernel
COUNTS = [[1], [1, 0, 31, 32, 33], [128, 129, 0, 256, 257, 1] + [0] * 4, [512, 513, 545, 2, 1025] + [0] * 25, [3] * 170]
# over twice the average and over a round of tiles: dealt out by size (up to 256 groups), equals among them
SKEWED = [[20] * 20 + [1100] + [300, 20] + [7, 0, 31] * 16, [130, 0] * 30 + [900, 140, 900], [2] * 150 + [700] + [2] * 149]


def offsets(counts):
    return torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32)


def close(out, ref):
    # one bf16 rounding of fp32 sums taken in another order: half an ulp (2^-9), and as much again where the rounding
    # of an operand of the following operation flipped; sums near zero by the size of their terms
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=2 ** -6, atol=2e-3)
    assert (out.cpu() != ref).float().mean() < 0.01


@pytest.mark.parametrize("counts", COUNTS + SKEWED)
@pytest.mark.parametrize("N,Kd", [(256, 1024), (768, 1152)])
def test_pair_plain(counts, N, Kd):
    g = torch.Generator().manual_seed(len(counts) + N)
    a = torch.randn(sum(counts), Kd, generator=g).to(torch.bfloat16)
    w = (torch.randn(len(counts), N, Kd, generator=g) * 0.05).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = moe_grouped_gemm(a.to(DEV), w.to(DEV), offsets(counts).to(DEV), status=status)
    assert status.item() == 0
    close(out, O.grouped_gemm(a, w, offsets(counts).long()))


@pytest.mark.parametrize("counts", COUNTS + SKEWED)
@pytest.mark.parametrize("inter,H", [(128, 128), (384, 640)])
def test_pair_swiglu_and_gather(counts, inter, H):
    E, S = len(counts), sum(counts)
    g = torch.Generator().manual_seed(len(counts) + inter)
    x = torch.randn(S, H, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, 2 * inter, H, generator=g) * 0.05).to(torch.bfloat16)
    perm = torch.randperm(S, generator=g).to(torch.int32)
    rows = x[perm.long()]
    off = offsets(counts)
    ref = torch.zeros(S, inter, dtype=torch.bfloat16)
    for e in range(E):
        s, t = int(off[e]), int(off[e + 1])
        gate, up = (rows[s:t].float() @ w[e].float().T).to(torch.bfloat16).split(inter, dim=1)
        ref[s:t] = torch.nn.functional.silu(gate) * up
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    plain = moe_grouped_swiglu(rows.to(DEV), w.to(DEV), off.to(DEV), status=status)
    gathered = moe_grouped_swiglu_gather(x.to(DEV), perm.to(DEV), 1, w.to(DEV), off.to(DEV), status=status)
    assert status.item() == 0
    close(plain, ref)
    assert torch.equal(plain, gathered)


@pytest.mark.parametrize("counts", [[40, 0, 300, 129, 17, 1], [3, 300, 128, 0, 60, 33] * 8])
def test_pair_shared_weights_and_partial_offsets(counts):
    """Groups that share weight sets (what ranks receive: source by source, the same experts again), offsets that start
    above 0 and end below the rows there are, a row table longer than the rows it lists."""
    E, inter, H, before, behind = 3, 256, 1024, 7, 50
    g = torch.Generator().manual_seed(len(counts))
    S = before + sum(counts) + behind
    off = offsets(counts) + before
    x = torch.randn(S, H, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, 2 * inter, H, generator=g) * 0.05).to(torch.bfloat16)
    perm = torch.randperm(S, generator=g).to(torch.int32)
    rows = x[perm.long()]
    ref, plain_ref = torch.zeros(S, inter, dtype=torch.bfloat16), torch.zeros(S, 2 * inter, dtype=torch.bfloat16)
    for i in range(len(counts)):
        s, t = int(off[i]), int(off[i + 1])
        plain_ref[s:t] = (rows[s:t].float() @ w[i % E].float().T).to(torch.bfloat16)
        gate, up = plain_ref[s:t].split(inter, dim=1)
        ref[s:t] = torch.nn.functional.silu(gate) * up
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = rows.to(DEV), w.to(DEV), off.to(DEV)
    plain = moe_grouped_gemm(*args, status=status)
    h = moe_grouped_swiglu(*args, status=status)
    gathered = moe_grouped_swiglu_gather(x.to(DEV), perm.to(DEV), 1, w.to(DEV), off.to(DEV), status=status)
    assert status.item() == 0
    lo, hi = int(off[0]), int(off[-1])
    for out in (plain, h):
        assert not out[:lo].any() and not out[hi:].any()
    close(plain[lo:hi], plain_ref[lo:hi])
    # gate, silu, up and their product may each fall one bf16 step apart (2^-7 of the value); below zero, where |silu'| is up
    # to 0.1, a step of the gate (2^-5 for |g| < 8) moves the product by 0.1 * 2^-5 * |u|, |u| < 8
    torch.testing.assert_close(h[lo:hi].cpu().float(), ref[lo:hi].float(), rtol=2 ** -5, atol=2.5e-2)
    assert (h[lo:hi].cpu() != ref[lo:hi]).float().mean() < 0.01
    assert torch.equal(gathered[lo:hi], h[lo:hi])
