"""GPU parity of the CTA-pair grouped GEMM (bf16, K % 128 == 0) at the edges of its tile shapes: 128 | 129 and 256 | 257
rows per expert, two tiles of up to 512 rows, tails of one row, one and an odd number of weight sub-tiles."""
import pytest
import torch

from mini_qwen_b200.kernels import moe_grouped_gemm, moe_grouped_swiglu
from mini_qwen_b200.kernels.moe_grouped_gemm import moe_grouped_swiglu_gather
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
COUNTS = [[1], [1, 0, 31, 32, 33], [128, 129, 0, 256, 257, 1], [512, 513, 545, 2, 1025], [3] * 170]


def offsets(counts):
    return torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32)


def close(out, ref):
    # one bf16 rounding of fp32 sums taken in another order: half an ulp (2^-9), and as much again where the rounding
    # of an operand of the following operation flipped; sums near zero by the size of their terms
    torch.testing.assert_close(out.cpu().float(), ref.float(), rtol=2 ** -6, atol=2e-3)
    assert (out.cpu() != ref).float().mean() < 0.01


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("N,Kd", [(256, 1024), (768, 1152)])
def test_pair_plain(counts, N, Kd):
    g = torch.Generator().manual_seed(len(counts) + N)
    a = torch.randn(sum(counts), Kd, generator=g).to(torch.bfloat16)
    w = (torch.randn(len(counts), N, Kd, generator=g) * 0.05).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = moe_grouped_gemm(a.to(DEV), w.to(DEV), offsets(counts).to(DEV), status=status)
    assert status.item() == 0
    close(out, O.grouped_gemm(a, w, offsets(counts).long()))


@pytest.mark.parametrize("counts", COUNTS)
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
