"""Rows of a grouped GEMM's result that no group covers are zero, whatever the buffer held: before the first offset
and behind the last; offsets of 16, 32 and 64 bits, rows of whole and of odd numbers of 16-byte pieces."""
import pytest
import torch

from mini_qwen_b200.kernels import moe_grouped_gemm

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("off", [[0, 3, 40, 40, 70], [5, 5, 30, 31, 33], [0, 0, 0, 0, 0], [10, 20, 20, 30, 69], [0, 70, 70, 70, 70]])
@pytest.mark.parametrize("wide", [torch.int64, torch.int32, torch.int16])
@pytest.mark.parametrize("dtype,N", [(torch.bfloat16, 256), (torch.float32, 33), (torch.float16, 5)])
def test_uncovered_rows_are_zero(off, wide, dtype, N):
    S, Kd, E = 70, 128, 4
    g = torch.Generator().manual_seed(N)
    a = torch.randn(S, Kd, generator=g).to(dtype)
    w = torch.randn(E, N, Kd, generator=g).to(dtype)
    covered = torch.zeros(S, dtype=torch.bool)
    covered[off[0]:off[E]] = True
    junk = [torch.full((S, N), 7.0, dtype=dtype, device=DEV) for _ in range(4)]
    del junk                                             # the allocator hands the result this memory
    offsets = torch.tensor(off, dtype=wide, device=DEV)
    a, w = a.to(DEV), w.to(DEV)
    out = moe_grouped_gemm(a, w, offsets)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    assert torch.equal(out, moe_grouped_gemm(a, w, offsets, status=status)) and status.item() == 0
    assert not out[~covered.to(DEV)].any()
    for e in range(E):
        s, t = off[e], off[e + 1]
        want = a[s:t].double() @ w[e].double().T
        # K fp32 products and sums, one rounding of the result (bf16: 2^-9)
        torch.testing.assert_close(out[s:t].double(), want, rtol=2 ** -7, atol=1e-4 * Kd)
