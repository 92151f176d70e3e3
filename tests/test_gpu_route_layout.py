"""The two layouts of the small-batch routing launch (csrc/router.cu), told apart by their bits: an input off the
16-byte grid always goes by expert, with the same order of the sums as one on it."""
import pytest
import torch

from mini_qwen_b200.kernels.moe_router import moe_route_small

pytestmark = pytest.mark.gpu
DEV = "cuda"


def off_grid(x):
    flat = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    flat[1:] = x.reshape(-1)
    return flat[1:].view(x.shape)


def probabilities(x, w, K):
    """Unnormalised softmax weights of the K chosen experts, in the order of the ids."""
    ids, weights = moe_route_small(x, w, K, renormalize=False)[:2]
    ids, order = ids.sort(dim=1)
    return ids, weights.gather(1, order)


@pytest.mark.parametrize("E", [8, 16, 32])
@pytest.mark.parametrize("T", [1, 4, 16])
def test_16_bit_batches_of_up_to_16_tokens_go_by_expert(E, T):
    g = torch.Generator(device=DEV).manual_seed(E + T)
    w = torch.randn(E, 2048, generator=g, device=DEV).to(torch.bfloat16) * 0.05
    for _ in range(8):
        x = torch.randn(T, 2048, generator=g, device=DEV).to(torch.bfloat16)
        for a, b in zip(probabilities(x, w, E), probabilities(off_grid(x), w, E)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("T,E,H", [(4, 8, 512), (16, 32, 512), (17, 32, 1024), (64, 16, 256), (64, 32, 2048)])
def test_fp32_sums_by_token_are_as_exact_as_by_expert(T, E, H):
    """Log-probabilities of all experts against fp64: the root mean square error by token is at most a tenth over the one
    by expert (both add eight products in a row and the rest in trees of the same depth; the samples scatter)."""
    g = torch.Generator(device=DEV).manual_seed(H)
    err = [0.0, 0.0]
    for _ in range(24):
        w = torch.randn(E, H, generator=g, device=DEV) * 0.1
        x = torch.randn(T, H, generator=g, device=DEV)
        exact = torch.log_softmax(x.double() @ w.double().T, dim=1)
        for i, rows in enumerate((x, off_grid(x))):
            ids, p = probabilities(rows, w, E)
            assert torch.equal(ids, torch.arange(E, device=DEV, dtype=ids.dtype).expand(T, E))
            err[i] += float((p.double().log() - exact).square().sum())
    assert err[0] ** 0.5 <= 1.1 * err[1] ** 0.5, err
