"""The W4A16 tile kernel for prefill-size groups (csrc/w4a16_tile.cu): single linears and grouped projections at the
edges of its tiles (rows 9 to 129 around the 16-row steps and the 128-row tile, columns that end inside a tile or after
the first of a pair, one and several quantisation groups, empty experts), with contiguous and with gathered rows, and
with several tiles to a CTA.  Where a call has too few rows for the kernel to pay, the dispatch sends it elsewhere: groups of
few rows are tested beside large ones.

Single linears are held to the fp32 result of the oracle's formula: the kernel multiplies exact integers q - z and adds
fp32 sums, so only the summation order (about 2^-22 of the sum of magnitudes) and the final rounding to bf16 (2^-9
relative) can differ.  The grouped projections are held to cases.w4_output_bar."""
import pytest
import torch

import cases
from mini_qwen_b200 import Qwen3MoEConfig, _cabi, synthetic
from mini_qwen_b200.kernels import moe_permute_plan
from mini_qwen_b200.kernels.moe_permute import gather_rows
from mini_qwen_b200.kernels.w4a16_gemm import (w4a16_gemm, w4a16_grouped_gemm, w4a16_grouped_swiglu,
                                               w4a16_grouped_swiglu_gather)
from mini_qwen_b200.model.layers import LinearW4A16, Qwen3MoEBlock
from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("M,K,N", [(9, 128, 32), (16, 256, 128), (17, 384, 96), (127, 128, 160), (128, 512, 256),
                                   (129, 256, 384), (300, 128, 4096), (2500, 256, 640),
                                   # two tiles to a CTA: 128 columns each with an odd number of groups; 256 columns
                                   # with a last pair that ends inside its first or second half or between them
                                   (4100, 384, 1024), (4100, 384, 2080), (4100, 384, 2176), (4100, 256, 2208)])
def test_single_linear_at_the_edges_of_the_tiles(M, K, N):
    g = torch.Generator().manual_seed(M + K + N)
    w = torch.randn(K, N, generator=g) * 0.05
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    qw, sc, qz = O.minmax_quantize(w, 128)
    got = w4a16_gemm(x.to(DEV), qw.contiguous().to(DEV), sc.to(DEV), qz.to(DEV), 128).cpu().double()
    ref = O.w4a16_linear(x, qw, sc, qz, 128, torch.float64).double()      # exact sums, rounded to bf16
    q = torch.stack([(qw >> (4 * i)) & 15 for i in range(8)], 1).reshape(K, N).double()
    z = torch.stack([(qz >> (4 * i)) & 15 for i in range(8)], 2).reshape(K // 128, N).double()
    dq = (q - z.repeat_interleave(128, 0)) * sc.double().repeat_interleave(128, 0)
    terms = x.double().abs() @ dq.abs()                                    # sum of magnitudes
    # one bf16 step (two roundings of neighbouring fp32 values may fall apart by one) and the fp32 summation error
    bound = 2.0 ** -7 * ref.abs() + 2.0 ** -20 * terms
    assert bool(((got - ref).abs() <= bound).all())


def dev_set(p):
    return tuple(t.to(DEV) for t in (p.qweight, p.scales.to(torch.bfloat16), p.qzeros))


@pytest.mark.parametrize("T,H,E,K,I,hot", [(37, 128, 4, 2, 32, 0), (65, 256, 4, 2, 160, 0), (200, 256, 8, 4, 384, 2),
                                           (300, 640, 6, 2, 128, 1)])
def test_grouped_projections_match_the_oracle(T, H, E, K, I, hot):
    """``hot`` experts take every token (groups of several tiles) and the last expert none."""
    lay = synthetic.w4a16_layer(T + I, T, H, E, K, I, group=128) if I % 128 == 0 else None
    g = torch.Generator().manual_seed(T)
    if lay is None:        # I that is no multiple of the quantisation group: gate/up only
        gate, up = synthetic._w4_proj(g, E, H, I, 128), synthetic._w4_proj(g, E, H, I, 128)
        x, down = torch.randn(T, H, generator=g).to(torch.bfloat16), None
    else:
        gate, up, down, x = lay.gate, lay.up, lay.down, lay.x
    ids = torch.stack([torch.cat([torch.arange(hot), hot + torch.randperm(E - 1 - hot, generator=g)[:K - hot]])
                       for _ in range(T)]).to(torch.int32).to(DEV)
    perm, _, off32, _ = moe_permute_plan(ids, E, want_int64_offsets=False)
    xd = x.to(DEV)
    rows = gather_rows(xd, perm, K)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    h = w4a16_grouped_swiglu_gather(xd, perm, K, dev_set(gate), dev_set(up), off32, status=status)
    plain = w4a16_grouped_swiglu(rows, dev_set(gate), dev_set(up), off32)
    if _cabi.load().mq_w4a16_tile_pays(T * K, E, I, H, 128, 1, 0):
        assert torch.equal(plain, h)
    off, sets = off32.cpu(), tuple((p.qweight, p.scales.to(torch.bfloat16), p.qzeros) for p in (gate, up))
    h32, h64 = (cases.w4_grouped_reference(rows.cpu(), sets, off, t) for t in (torch.float32, torch.float64))
    cases.w4_output_bar(h.cpu(), h32, h64)
    cases.w4_output_bar(plain.cpu(), h32, h64)
    if down is not None:
        o = w4a16_grouped_gemm(h, *dev_set(down), off32)
        dset = ((down.qweight, down.scales.to(torch.bfloat16), down.qzeros),)
        o32, o64 = (cases.w4_grouped_reference(h.cpu(), dset, off, t) for t in (torch.float32, torch.float64))
        cases.w4_output_bar(o.cpu(), o32, o64)
    assert status.item() == 0


@pytest.mark.parametrize("N,K", [(32, 128), (128, 256), (96, 384), (160, 128)])
def test_plain_projection_of_small_groups_beside_a_large_one(N, K):
    g = torch.Generator().manual_seed(N + K)
    counts = [9, 16, 0, 17, 1, 15, 1200]
    off = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32)
    S, E = int(off[-1]), len(counts)
    assert _cabi.load().mq_w4a16_tile_pays(S, E, N, K, 128, 0, 0)
    p = synthetic._w4_proj(g, E, K, N, 128)
    x = torch.randn(S, K, generator=g).to(torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = w4a16_grouped_gemm(x.to(DEV), *dev_set(p), off.to(DEV), status=status).cpu()
    sets = ((p.qweight, p.scales.to(torch.bfloat16), p.qzeros),)
    r32, r64 = (cases.w4_grouped_reference(x, sets, off, t) for t in (torch.float32, torch.float64))
    cases.w4_output_bar(got, r32, r64)
    assert status.item() == 0


def test_several_tiles_to_a_cta_and_groups_that_share_weights():
    """More tiles than the CTAs take in two rounds, groups of 0 to over 1000 rows, twice as many groups as weight sets,
    offsets that start above 0 and end below the rows there are."""
    T, K, H, E, I = 700, 8, 384, 6, 1024
    g = torch.Generator().manual_seed(3)
    gate, up = synthetic._w4_proj(g, E, H, I, 128), synthetic._w4_proj(g, E, H, I, 128)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    counts = torch.tensor([5, 0, 1, 16, 17, 127, 128, 129, 1100, 300, 0, 2100, 1650])       # the first: in no group
    off = counts.cumsum(0).to(torch.int32)
    lo, hi = int(off[0]), int(off[-1])
    assert hi < T * K
    perm = torch.randperm(T * K, generator=g).to(torch.int32).to(DEV)
    rows = gather_rows(x, perm, K)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    h = w4a16_grouped_swiglu_gather(x, perm, K, dev_set(gate), dev_set(up), off.to(DEV), status=status)
    plain = w4a16_grouped_swiglu(rows, dev_set(gate), dev_set(up), off.to(DEV))
    assert torch.equal(plain[lo:hi], h[lo:hi]) and not plain[:lo].any() and not plain[hi:].any()
    sets = tuple((p.qweight, p.scales.to(torch.bfloat16), p.qzeros) for p in (gate, up))
    h32, h64 = (cases.w4_grouped_reference(rows.cpu(), sets, off, t) for t in (torch.float32, torch.float64))
    cases.w4_output_bar(h[lo:hi].cpu(), h32[lo:hi], h64[lo:hi])
    o = w4a16_grouped_gemm(rows, *dev_set(gate), off.to(DEV))
    assert not o[:lo].any() and not o[hi:].any()
    o32, o64 = (cases.w4_grouped_reference(rows.cpu(), sets[:1], off, t) for t in (torch.float32, torch.float64))
    cases.w4_output_bar(o[lo:hi].cpu(), o32[lo:hi], o64[lo:hi])
    assert status.item() == 0


@pytest.mark.parametrize("counts,E", [((9, 11, 10), 3), ([8, 9, 8] * 133 + [30], 8)])
def test_swiglu_keeps_the_exact_quotient_where_the_stream_kernel_did_not_run(counts, E):
    """Fewer than 32 rows, and more than 384 groups: silu with expf and a true quotient, i.e. torch's own silu of the
    bf16 gate, bit for bit (an approximation falls to the other bf16 neighbour once in about 2^11 elements)."""
    H, I = 256, 2048 if E == 3 else 256
    g = torch.Generator().manual_seed(E)
    gate, up = (dev_set(synthetic._w4_proj(g, E, H, I, 128)) for _ in range(2))
    off = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    S = int(off[-1])
    assert S > 8 * len(counts)
    x = (torch.randn(S, H, generator=g) * 0.3).to(torch.bfloat16).to(DEV)
    # the projections by themselves, in the same order of the sums: each group's rows forty times over, so that the plain
    # call pays on the tile kernel, which keeps the rows of a group apart
    many = torch.cat([x[s:t].repeat(40, 1) for s, t in zip(off.tolist(), off.tolist()[1:])])
    first = torch.cat([40 * s + torch.arange(t - s) for s, t in zip(off.tolist(), off.tolist()[1:])]).to(DEV)
    gate_rows, up_rows = (w4a16_grouped_gemm(many, *w, off * 40)[first] for w in (gate, up))
    want = torch.nn.functional.silu(gate_rows) * up_rows
    perm = torch.arange(S, dtype=torch.int32, device=DEV)
    assert torch.equal(w4a16_grouped_swiglu_gather(x, perm, 1, gate, up, off), want)
    direct = w4a16_grouped_swiglu(x, gate, up, off)
    if E == 3:                     # goes to the cp.async kernel, as its projections do
        want = torch.nn.functional.silu(w4a16_grouped_gemm(x, *gate, off)) * w4a16_grouped_gemm(x, *up, off)
    assert torch.equal(direct, want)


def test_gather_entry_point_rejects_what_the_kernel_does_not_cover():
    x = torch.zeros(4, 128, dtype=torch.bfloat16, device=DEV)
    w = tuple(t.to(DEV) for t in (torch.zeros(1, 16, 40, dtype=torch.int32), torch.zeros(1, 1, 40, dtype=torch.bfloat16),
                                  torch.zeros(1, 1, 5, dtype=torch.int32)))
    perm = torch.arange(4, dtype=torch.int32, device=DEV)
    off = torch.tensor([0, 4], dtype=torch.int32, device=DEV)
    with pytest.raises(ValueError):
        w4a16_grouped_swiglu_gather(x, perm, 1, w, w, off)                 # 40 columns: not a multiple of 32


def test_expected_rows_choose_the_kernel_and_nothing_else():
    """A buffer of 512 rows of which 64 lie in the 16 groups (decode by replication over eight ranks): with that said the
    call runs on the cp.async kernel, told apart by its bits (which zero points off the 16-byte grid force)."""
    E, H, I, S = 16, 4096, 1024, 512                     # wide enough for the order of the sums to show in some bf16 bit
    g = torch.Generator().manual_seed(9)
    qw, sc, qz = dev_set(synthetic._w4_proj(g, E, I, H, 128))
    flat = torch.empty(qz.numel() + 1, dtype=torch.int32, device=DEV)
    flat[1:] = qz.reshape(-1)
    off_grid = (qw, sc, flat[1:].view(qz.shape))
    x = torch.randn(S, I, generator=g).to(torch.bfloat16).to(DEV)
    off = (100 + 4 * torch.arange(E + 1)).to(torch.int32).to(DEV)
    streamed, told, untold = (w4a16_grouped_gemm(x, *w, off, rows=r) for w, r in ((off_grid, 0), ((qw, sc, qz), 64), ((qw, sc, qz), 0)))
    assert torch.equal(told, streamed) and not torch.equal(untold, streamed)
    assert float((told.float() - untold.float()).norm() / untold.float().norm()) < 2 ** -9


class Recorder:
    """The library, with the arguments of every call kept."""

    def __init__(self, lib):
        self.lib, self.calls = lib, []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return getattr(self.lib, name)(*args)
        return call


def test_every_launch_of_the_kernel_has_a_status_word(monkeypatch):
    """The kernel leaves part of its result unwritten when a bounded wait runs out; check_status() must be able to say
    so.  (No wait is made to run out here: the word is set by hand.)"""
    spy = Recorder(_cabi.load())
    monkeypatch.setattr(_cabi, "load", lambda: spy)
    lin = LinearW4A16(256, 128).to(DEV)
    x = torch.randn(200, 256, device=DEV).to(torch.bfloat16)
    lin(x[:8])
    lin.check_status()
    lin(x)
    lin(x.reshape(2, 100, 256))
    launches = [a for n, a in spy.calls if n == "mq_w4a16_linear_ex"]
    assert [a[-2] for a in launches] == [None, lin._status.data_ptr(), lin._status.data_ptr()]
    lin.check_status()
    lin._status.fill_(1)
    with pytest.raises(RuntimeError):
        lin.check_status()
    assert set(lin.state_dict()) == {"qweight", "scales", "qzeros"}

    cfg = Qwen3MoEConfig(hidden_size=256, intermediate_size=128, num_experts=8, num_experts_per_tok=2)
    blk = Qwen3MoEBlock.from_stacked_w4(cfg, torch.randn(8, 256, device=DEV).to(torch.bfloat16),
                                        *synthetic.w4a16_stacks_on_device(DEV, 3, 8, 256, 128))
    for kernel in ("stream", "mma"):
        spy.calls.clear()
        blk.w4_kernel = kernel
        blk._forward_staged(x)
        word = blk._status.data_ptr()
        seen = [n for n, a in spy.calls if n.startswith("mq_w4a16_grouped") and word in a]
        assert len(seen) == 2 and all(word in a for n, a in spy.calls if n.startswith("mq_w4a16_grouped")), spy.calls
    blk.check_status()
