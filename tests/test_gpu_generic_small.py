"""The small-group kernel of csrc/grouped_gemm_generic.cu at the edges of its tiles (16 rows, 32 columns, 128 k), with
and without vector loads, against fp64 sums.  fp32: a sum of Kd fp32 products may be off by Kd * 2^-24 of the sum of
their magnitudes; 16-bit types add one rounding of the result."""
import pytest
import torch

from mini_qwen_b200.kernels import moe_grouped_gemm, moe_grouped_swiglu

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,N,Kd", [((1, 0, 15), 31, 4), ((16, 17, 1), 32, 127), ((32, 3, 0), 33, 128),
                                       ((7, 31, 2), 96, 260), ((20, 20, 20), 5, 129),
                                       # many groups: the fused call here, the plain one with 64-row tiles; then both so
                                       ((26,) * 128, 33, 20), ((30,) * 128, 33, 20)])
def test_small_groups(dtype, rows, N, Kd):
    if dtype != torch.float32 and Kd % 64 == 0 and N % 128 == 0:
        pytest.skip("the tcgen05 kernel takes this shape")
    g = torch.Generator().manual_seed(sum(rows) + N + Kd)
    S, E = sum(rows), len(rows)
    off = torch.tensor([sum(rows[:i]) for i in range(E + 1)], dtype=torch.int32)
    a = torch.randn(S, Kd, generator=g).to(dtype)
    w = torch.randn(E, N, Kd, generator=g).to(dtype)
    w2 = torch.randn(E, 2 * N, Kd, generator=g).to(dtype) * 0.1
    got = moe_grouped_gemm(a.to(DEV), w.to(DEV), off.to(DEV)).cpu().double()
    h = moe_grouped_swiglu(a.to(DEV), w2.to(DEV), off.to(DEV)).cpu().double()
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
    for e in range(E):
        lo, hi = int(off[e]), int(off[e + 1])
        x = a[lo:hi].double()
        ref, terms = x @ w[e].double().T, x.abs() @ w[e].double().abs().T
        assert bool(((got[lo:hi] - ref).abs() <= ulp * ref.abs() + Kd * 2.0 ** -24 * terms).all())
        gate, up = x @ w2[e, :N].double().T, x @ w2[e, N:].double().T
        tg, tu = x.abs() @ w2[e, :N].double().abs().T, x.abs() @ w2[e, N:].double().abs().T
        sum_err = Kd * 2.0 ** -24
        # four roundings (gate, silu, up, product), and the sums' errors: |silu'| <= 1.1
        want = gate / (1 + torch.exp(-gate)) * up
        bound = 4 * ulp * (want.abs() + gate.abs() * up.abs()) + 1.1 * sum_err * tg * up.abs() + sum_err * tu * gate.abs() + 1e-6
        assert bool(((h[lo:hi] - want).abs() <= bound).all())
