"""CPU checks of the host side: int4 format, quantiser, LinearW4A16 constructors, the module tree
of the block, and that libmqmoe.so loads and exports every symbol include/mqmoe.h declares.
No kernel is launched here."""
import ctypes
import os
import re

import pytest
import torch
import torch.nn as nn

import cases
from mini_qwen_b200 import Qwen3MoEConfig, _cabi
from mini_qwen_b200.kernels import moe_grouped_gemm, moe_permute, moe_router, moe_unpermute, w4a16_gemm
from mini_qwen_b200.model.layers import LinearW4A16, Qwen3MoEBlock, RMSNorm
from mini_qwen_b200.quantization import _per_group_minmax_quantize, pack_int4, quantize_awq, unpack_int4
from oracle import moe_oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pack_unpack_roundtrip_along_k():
    # reference: tests/test_w4a16_gemm.py:67-75
    K, N = 128, 64
    w = torch.randint(0, 16, (K, N), dtype=torch.int32, generator=torch.Generator().manual_seed(0))
    packed = pack_int4(w.T).T
    assert packed.shape == (K // 8, N) and packed.dtype == torch.int32
    assert torch.equal(unpack_int4(packed.T).T, w)


def test_pack_unpack_roundtrip_along_n():
    # reference: tests/test_w4a16_gemm.py:78-84
    z = torch.randint(0, 16, (8, 64), dtype=torch.int32, generator=torch.Generator().manual_seed(1))
    packed = pack_int4(z)
    assert packed.shape == (8, 8)
    assert torch.equal(unpack_int4(packed), z)


def test_pack_layout_and_sign():
    x = torch.tensor([[1, 2, 3, 4, 5, 6, 7, 8]], dtype=torch.int32)
    assert pack_int4(x).item() == 0x87654321 - (1 << 32)     # nibble 7 >= 8 -> negative int32
    assert torch.equal(pack_int4(x), O.pack_int4(x))
    with pytest.raises(AssertionError):
        pack_int4(torch.zeros(3, 7, dtype=torch.int32))


def test_minmax_quantiser_matches_oracle():
    w = torch.randn(256, 64, generator=torch.Generator().manual_seed(2))
    for a, b in zip(_per_group_minmax_quantize(w, 128), O.minmax_quantize(w, 128)):
        assert torch.equal(a, b)
    with pytest.raises(AssertionError):
        _per_group_minmax_quantize(torch.randn(100, 64), 128)
    with pytest.raises(NotImplementedError):
        quantize_awq(None, None)


def test_from_gptq_zero_plus_one_clamps():
    g = cases.golden("quant_cases")
    stored = pack_int4(torch.arange(16, dtype=torch.int32).reshape(1, 16))
    layer = LinearW4A16.from_gptq(torch.zeros(16, 16, dtype=torch.int32), stored, torch.ones(1, 16) * 0.0123)
    assert torch.equal(layer.qzeros, torch.from_numpy(g["gptq_zeros"]))
    assert torch.equal(layer.scales, cases.from_bits(g["gptq_scales"], torch.bfloat16))
    assert unpack_int4(layer.qzeros)[0, -2:].tolist() == [15, 15]      # stored 14 -> 15, stored 15 stays 15
    raw = LinearW4A16.from_gptq(torch.zeros(16, 16, dtype=torch.int32), stored, torch.ones(1, 16), zero_plus_one=False)
    assert torch.equal(raw.qzeros, stored)


def test_from_float_shapes_and_state_dict_keys():
    lin = nn.Linear(256, 64, bias=False)
    q = LinearW4A16.from_float(lin, group_size=128)
    assert q.qweight.shape == (32, 64) and q.scales.shape == (2, 64) and q.qzeros.shape == (2, 8)
    assert set(q.state_dict()) == {"qweight", "scales", "qzeros"}
    qw, sc, qz = O.minmax_quantize(lin.weight.data.float().T.contiguous(), 128)
    assert torch.equal(q.qweight, qw) and torch.equal(q.scales, sc) and torch.equal(q.qzeros, qz)


def test_block_module_tree_matches_hf_names():
    cfg = Qwen3MoEConfig(hidden_size=32, intermediate_size=16, num_experts=4, num_experts_per_tok=2)
    blk = Qwen3MoEBlock(cfg)
    keys = set(blk.state_dict())
    assert "gate.weight" in keys
    for e in range(4):
        for p in ("gate_proj", "up_proj", "down_proj"):
            assert f"experts.{e}.{p}.weight" in keys
    assert blk.num_experts == 4 and blk.num_experts_per_tok == 2 and blk.norm_topk_prob is True
    # stacking keeps the per-expert tensors addressable and shares their storage
    before = {k: v.clone() for k, v in blk.state_dict().items()}
    blk.finalize()
    for k, v in blk.state_dict().items():
        assert torch.equal(v, before[k])
    assert blk.experts[1].up_proj.weight.data_ptr() == blk._stacks["w13"][1, 16:].data_ptr()
    # an in-place load writes through to the stacks
    blk.load_state_dict({k: torch.full_like(v, 0.5) for k, v in before.items()})
    assert float(blk._stacks["w2"].min()) == 0.5
    # replacing a projection invalidates the stacks
    epoch = blk._epoch[0]
    blk.experts[0].gate_proj = nn.Linear(32, 16, bias=False)
    assert blk._epoch[0] == epoch + 1


def test_block_quantize_to_w4a16_swaps_modules():
    cfg = Qwen3MoEConfig(hidden_size=64, intermediate_size=32, num_experts=2, num_experts_per_tok=1)
    blk = Qwen3MoEBlock(cfg)
    blk.quantize_to_w4a16(group_size=32)
    assert all(isinstance(getattr(ex, p), LinearW4A16) for ex in blk.experts for p in ("gate_proj", "up_proj", "down_proj"))
    blk.finalize()
    assert blk._stacks["w4"] and blk._stacks["gate_proj"][0].shape == (2, 8, 32)
    assert blk.experts[1].down_proj.qweight.data_ptr() == blk._stacks["down_proj"][0][1].data_ptr()


def test_library_exports_every_declared_symbol():
    header = open(os.path.join(ROOT, "include", "mqmoe.h")).read()
    declared = set(re.findall(r"\b(mq_[a-z0-9_]+)\s*\(", header))
    declared -= {"mq_status", "mq_dtype"}
    assert declared == set(_cabi.PROTOTYPES), declared ^ set(_cabi.PROTOTYPES)
    lib = _cabi.load()
    for name in declared:
        assert isinstance(getattr(lib, name), ctypes._CFuncPtr)
    assert lib.mq_version() >= 1
    assert lib.mq_status_string(2).decode().startswith("size outside")


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    monkeypatch.setattr(_cabi, "_lib", None)
    monkeypatch.setenv("MQMOE_LIB", str(tmp_path / "nope.so"))
    with pytest.raises(RuntimeError, match="no CPU or PyTorch fallback"):
        _cabi.load()


def test_cpu_tensors_are_rejected():
    x = torch.randn(4, 32)
    with pytest.raises(ValueError, match="CUDA"):
        moe_router(x, torch.randn(8, 32), 2)
    with pytest.raises(ValueError, match="CUDA"):
        moe_permute(x, torch.zeros(4, 2, dtype=torch.int64), 8)
    with pytest.raises(ValueError, match="CUDA"):
        moe_grouped_gemm(x, torch.randn(8, 16, 32), torch.zeros(9, dtype=torch.int64))
    with pytest.raises(ValueError, match="CUDA"):
        moe_unpermute(torch.randn(8, 32), torch.rand(4, 2), torch.zeros(4, 2, dtype=torch.int64), 4)
    with pytest.raises(AssertionError):
        w4a16_gemm(x.to(torch.bfloat16), torch.zeros(4, 8, dtype=torch.int32),
                   torch.zeros(1, 8, dtype=torch.bfloat16), torch.zeros(1, 1, dtype=torch.int32), 32)


def test_argument_checks_return_status_without_a_gpu():
    lib = _cabi.load()
    # nothing is launched when the argument check fails, so these are safe on a CPU-only host
    assert lib.mq_router_topk(None, 0, None, 0, None, 4, 32, 8, 9, 0, None, 0, None, None, None, None) == 2   # K > E
    assert lib.mq_router_topk(None, 0, None, 0, None, 4, 32, 8, 2, 0, None, 0, None, None, None, None) == 1   # null
    assert lib.mq_router_topk(None, 7, None, 0, None, 4, 32, 8, 2, 0, None, 0, None, None, None, None) == 1   # dtype
    assert lib.mq_permute_plan(None, 1, 4, 2, 128, None, None, None, None, None, 0, None) == 1             # no offsets
    assert lib.mq_permute_plan(None, 1, 4, 2, 2048, None, None, None, None, None, 0, None) == 2            # E > 1024
    assert lib.mq_w4a16_grouped_gemm(None, None, None, None, None, 4, 1, 1, 8, 128, 48, None, None) == 2      # group % 32
    assert lib.mq_unpermute_combine(None, 1, None, None, 4, 33, 64, None, None) == 2                        # K > 32
    assert lib.mq_permute_workspace_bytes(131072, 128) >= 64 * 128 * 4


def test_from_stacked_shares_storage():
    cfg = Qwen3MoEConfig(hidden_size=32, intermediate_size=16, num_experts=4, num_experts_per_tok=2)
    w13, w2, r = torch.randn(4, 32, 32), torch.randn(4, 32, 16), torch.randn(4, 32)
    blk = Qwen3MoEBlock.from_stacked(cfg, r, w13, w2)
    assert blk.experts[2].up_proj.weight.data_ptr() == w13[2, 16:].data_ptr()
    assert torch.equal(blk.state_dict()["experts.3.down_proj.weight"], w2[3])
    assert blk._ready()["w13"].data_ptr() == w13.data_ptr()       # no restack needed


def test_static_router_scratch_covers_every_batch_up_to_16384_tokens():
    """mq_router_topk_static promises room for any batch up to 16384 tokens at the Qwen3-30B-A3B router
    shape.  The request is not monotonic in T (the logits are kept in several K slices for small
    batches), so every T is checked against the 10 MiB array, and the first refused batch size is pinned."""
    lib = _cabi.load()
    limit = 10 << 20
    worst = max(lib.mq_router_workspace_bytes(T, 2048, 128) for T in range(1, 16385))
    assert worst <= limit, worst
    assert worst == 2 * 9440 * 128 * 4                  # the documented peak: two slices at 9440 tokens
    assert lib.mq_router_workspace_bytes(20480, 2048, 128) == limit     # the largest batch that fits
    # one token more is refused by the argument check, before anything touches a device
    assert lib.mq_router_topk_static(None, 1, None, 1, None, 20481, 2048, 128, 8, 0, None, None, None, None) == 6


def test_ep_entry_points_reject_bad_poll_budgets_without_a_gpu():
    lib = _cabi.load()
    assert lib.mq_ep_barrier(None, None, 2, 0, 0, None, None) == 1                  # null pointers
    assert lib.mq_stack_tensors(None, 3, 64, 1, None, None) == 1                     # null pointers
    assert lib.mq_stack_tensors(None, 0, 64, 1, None, None) == 0                     # nothing to do
    assert lib.mq_stack_tensors(None, 70000, 64, 1, None, None) == 1


def test_decode_replication_entry_points_reject_bad_arguments_without_a_gpu():
    lib = _cabi.load()
    assert lib.mq_ep_gather_tokens(None, 1, 4, 2048, 2, 0, None, None, None, 0, None, None) == 1     # null pointers
    assert lib.mq_ep_gather_tokens(None, 1, 4, 2048, 2, 2, None, None, None, 0, None, None) == 1     # rank >= G
    assert lib.mq_ep_gather_tokens(None, 1, 4, 2047, 2, 0, None, None, None, 0, None, None) == 2     # rows not 16-byte multiples
    # tokens must be G * T
    assert lib.mq_ep_send_partials(None, 1, None, None, None, 9, 8, 2048, 4, 2, 0, 64, None, None, None, None, 0,
                                   None, None) == 1
    assert lib.mq_ep_send_partials(None, 1, None, None, None, 8, 33, 2048, 4, 2, 0, 64, None, None, None, None, 0,
                                   None, None) == 2                                             # K > 32
    assert lib.mq_ep_sum_partials(None, 1, None, 4, 2048, 2, None, None) == 1                        # null pointers
    assert lib.mq_ep_sum_partials(None, 1, None, 4, 2046, 2, None, None) == 2                        # H not a multiple of 4
    assert lib.mq_rms_norm(None, 1, None, 1e-6, 4, 2048, None, None) == 1                            # null pointers
    assert lib.mq_rms_norm(None, 1, None, 1e-6, 0, 2048, None, None) == 0                            # nothing to do
    assert lib.mq_unpermute_combine_residual(None, 1, None, None, None, 4, 33, 64, None, None) == 2  # K > 32


def _small_block(quantised=False):
    blk = Qwen3MoEBlock(Qwen3MoEConfig(hidden_size=64, intermediate_size=32, num_experts=2, num_experts_per_tok=1))
    if quantised:
        blk.quantize_to_w4a16(group_size=32)
    return blk


@pytest.mark.parametrize("quantised", [False, True])
@pytest.mark.parametrize("where", ["router", "expert", "weight_norm", "replica"])
def test_weights_that_their_modules_do_not_keep_under_their_own_name(quantised, where):
    """A parametrised router or expert projection, old-style weight norm, and the plain-attribute weights of a
    DataParallel replica: found through the attribute, and a router that is computed on access (whose address a
    description must not keep) goes stage by stage."""
    blk = _small_block(quantised)
    if where == "router":
        nn.utils.parametrize.register_parametrization(blk.gate, "weight", nn.Identity())
    elif where == "expert":
        nn.utils.parametrize.register_parametrization(blk.experts[0].gate_proj, "qweight" if quantised else "weight",
                                                      nn.Identity())
    elif where == "weight_norm":
        blk.gate = nn.utils.weight_norm(blk.gate)
    else:
        for m in blk.modules():
            for name, p in list(m._parameters.items()):
                if p is not None:
                    del m._parameters[name]
                    setattr(m, name, p.data)
    assert len(blk._sentinel()) == 2 and blk._ready() is blk._stacks
    assert blk._native_layer() is None                       # CPU tensors, or a router its module does not keep
    dt = torch.bfloat16 if quantised else torch.float32
    with pytest.raises((ValueError, AssertionError), match="CUDA"):
        blk(torch.zeros(3, 64, dtype=dt))                    # the error of CPU tensors, not a missing name


def test_linear_w4a16_with_a_parametrised_buffer():
    lin = LinearW4A16(64, 32, 32)
    nn.utils.parametrize.register_parametrization(lin, "scales", nn.Identity())
    with pytest.raises(AssertionError, match="CUDA"):
        lin(torch.zeros(3, 64, dtype=torch.bfloat16))


@pytest.mark.parametrize("what", ["plain", "hook", "global hook", "replica", "own forward"])
def test_half_layer_calls_a_norm_that_does_more_than_normalise(what):
    blk, norm = _small_block(), RMSNorm(64)
    native = []
    blk._forward_native = lambda h, residual, weight, eps: native.append(weight) or h
    blk.forward = lambda h, residual: "called"
    handle = None
    if what == "hook":
        norm.register_forward_hook(lambda m, i, o: None)
    elif what == "global hook":
        handle = nn.modules.module.register_module_forward_pre_hook(lambda m, i: None)
    elif what == "replica":
        w = norm._parameters.pop("weight").data
        norm.weight = w
    elif what == "own forward":
        norm.forward = lambda h: h
    h = torch.zeros(3, 64)
    try:
        if what == "plain":
            assert blk.half_layer(h, norm) is h and native == [norm.weight.data_ptr()]
        elif what == "own forward":
            assert blk.half_layer(h, norm) == "called" and not native
        else:
            with pytest.raises(ValueError, match="CUDA"):    # the norm itself ran, on CPU tensors
                blk.half_layer(h, norm)
            assert not native
    finally:
        if handle is not None:
            handle.remove()


@pytest.mark.parametrize("quantised", [False, True])
def test_finalize_drops_the_description_of_the_old_stacks(quantised):
    """A description holds the addresses of up to nine stacks; the two that are compared on each call may come out
    of the allocator where they were while the others have moved."""
    blk = _small_block(quantised)
    blk._native_layer()
    assert blk._native is not None
    blk.finalize()
    assert blk._native is None


def test_the_block_call_hands_its_status_word_to_every_kernel_that_has_bounded_waits():
    """In csrc/block.cu: each library call that takes a status word is given the caller's, and none is made in a form
    without one (mq_x where mq_x_ex has one)."""
    header = open(os.path.join(ROOT, "include", "mqmoe.h")).read()
    prototypes = dict(re.findall(r"\bint (mq_[a-z0-9_]+)\(([^;]*)\);", header))
    with_status = {n for n, args in prototypes.items() if "d_status" in args}
    without = {n for n in prototypes if n + "_ex" in with_status}
    source = open(os.path.join(ROOT, "mini-qwen-llm_b200", "csrc", "block.cu")).read()
    source = source[source.index('extern "C" int mq_moe_forward('):]
    calls = re.findall(r"MQ_BLOCK_STEP\((mq_[a-z0-9_]+)\((.*?)\)\);", source, flags=re.S)
    named = {n for n, _ in calls}
    assert {"mq_w4a16_grouped_gemm_ex", "mq_grouped_gemm"} <= named and not named & without
    for name, args in calls:
        assert name not in with_status or "d_status" in args, name


def test_zero_points_off_the_16_byte_grid_keep_a_layer_off_the_tile_kernel():
    """Views into a flat checkpoint buffer: the tile kernel copies zero points in bulk and refuses them, the others read
    them word by word.  The stream kernel's prepared rows show in the workspace."""
    lib = _cabi.load()
    L = _cabi.MoELayer(hidden=256, inter=128, experts=8, top_k=2, group_size=128, dtype=_cabi.MQ_BF16,
                       router_dtype=_cabi.MQ_BF16, renormalize=1)
    for name in ("gate", "up", "down"):
        for i in range(3):
            getattr(L, name)[i] = 4096
    T, rows = 200, 400
    tile = lib.mq_moe_forward_workspace_bytes(ctypes.addressof(L), T)
    L.down[2] = 4100
    assert lib.mq_moe_forward_workspace_bytes(ctypes.addressof(L), T) == tile
    for name in ("gate", "up"):
        getattr(L, name)[2] = 4100
        assert lib.mq_moe_forward_workspace_bytes(ctypes.addressof(L), T) >= tile + rows * 256 * 2
        getattr(L, name)[2] = 4096
    blk = _small_block(True)
    flat = torch.zeros(257, dtype=torch.int32)
    at = (-flat.data_ptr() // 4) % 4
    for off, want in ((at, True), (at + 1, False)):
        st = {"gate_proj": (torch.zeros(2, 16, 32), None, flat[off:]), "up_proj": (None, None, flat[at:]), "group_size": 128}
        assert blk._w4_tile(st, 1000) is want
        st["gate_proj"], st["up_proj"] = (st["gate_proj"][0], None, flat[at:]), (None, None, flat[off:])
        assert blk._w4_tile(st, 1000) is want


def test_expert_parallel_w4a16_calls_say_how_many_rows_are_a_ranks_own(monkeypatch):
    """Decode by replication hands over all ranks' slots, the peer path a buffer with room for them; the choice of the
    kernels goes by the slots that one rank's experts own on average."""
    from mini_qwen_b200.model.layers import moe
    T, K, E, G, H, I = 8, 2, 16, 4, 64, 32
    blk = Qwen3MoEBlock(Qwen3MoEConfig(hidden_size=H, intermediate_size=I, num_experts=E, num_experts_per_tok=K))
    blk.ep_size, blk.ep_rank, blk.num_local_experts = G, 1, E // G
    st = {"w4": True, "group_size": 32, "gate_proj": (), "up_proj": (), "down_proj": (torch.zeros(1),) * 3}
    seen = []

    class Peer:
        def gather_tokens(self, x):
            return x.repeat(G, 1)

        def recv_rows(self):
            return torch.zeros(G * T * K, H, dtype=torch.bfloat16)

        def __getattr__(self, name):
            return (lambda *a, **k: (None, None)) if name == "exchange_plan" else (lambda *a, **k: torch.zeros(1))
    blk._ensure_peer = lambda *a: Peer()
    blk._status_word = lambda device: torch.zeros(1, dtype=torch.int32)
    off = torch.arange(E + 1, dtype=torch.int32)
    monkeypatch.setattr(moe, "route_small_workspace", lambda *a: torch.zeros(1))
    monkeypatch.setattr(moe, "moe_route_small", lambda x, *a, **k: (None, None, None, None, off, x, x))
    monkeypatch.setattr(moe, "w4a16_stream_swiglu", lambda xp, *a, **k: xp)
    monkeypatch.setattr(moe, "w4a16_grouped_swiglu", lambda x, *a, **k: seen.append((x.shape[0], k["rows"])) or x)
    monkeypatch.setattr(moe, "w4a16_grouped_gemm", lambda x, *a, **k: seen.append((x.shape[0], k["rows"])) or x)
    x = torch.zeros(T, H, dtype=torch.bfloat16)
    blk._forward_replicated(x, st, T, K, E)
    assert seen == [(G * T, T * K)]
    seen.clear()
    blk._forward_peer(x, st, None, None, None, None, off, T, K, E)
    assert seen == [(G * T * K, T * K)] * 2


def test_which_kernel_a_w4a16_call_goes_to():
    """The rule by sizes at the places where both sides were measured (us, streaming kernels | tile kernel)."""
    pays = _cabi.load().mq_w4a16_tile_pays

    def fused(S, E, N, K, prepare=1):
        return pays(S, E, N, K, 128, 1, prepare)

    def one(S, E, N, K):
        return pays(S, E, N, K, 128, 0, 0)
    for tile, calls in ((0, [(232, 16, 128, 2048), (254, 8, 128, 1792), (116, 8, 256, 1536), (448, 16, 128, 2048),
                             (64, 1, 768, 2048), (100, 2, 384, 1024), (1024, 128, 768, 2048)]),   # 12|21 12|19 11|18 15|21 11|20 9|13
                        (1, [(1280, 128, 768, 2048), (2048, 128, 768, 2048), (32768, 128, 768, 2048), (160, 16, 768, 512),
                             (400, 16, 384, 1024), (520, 64, 384, 1024), (3000, 8, 768, 2048)])):  # 109|103 152|104 - 19|10 20|14
        for c in calls:
            assert fused(*c) == tile, c
    for tile, calls in ((0, [(9, 1, 512, 512), (16, 1, 4096, 512), (16, 1, 2048, 2048), (27, 3, 1024, 384),
                             (152, 16, 1280, 128), (1160, 128, 1536, 128), (1104, 128, 768, 256)]),
                        (1, [(17, 1, 512, 512), (17, 1, 2048, 4096), (33, 1, 512, 2048), (500, 1, 2048, 4096),
                             (160, 16, 2048, 768), (1280, 128, 2048, 768), (32768, 128, 2048, 768)])):
        for c in calls:
            assert one(*c) == tile, c
    assert fused(64, 16, 768, 2048) == 0 and one(64, 16, 2048, 768) == 0          # four rows a group: never
    # more groups than the stream kernel takes: the cp.async kernel is the alternative
    assert fused(8 * 400 + 1, 400, 768, 2048) == 1 and fused(8 * 400, 400, 768, 2048) == 0
    # sizes that the tile kernel does not take, and nonsense
    assert pays(4000, 4, 768, 2048, 64, 1, 0) == 0 and one(4000, 4, 100, 2048) == 0 and one(-1, 0, 0, 0) == 0
