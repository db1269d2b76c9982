"""A router's logits: a product with few rows, at the edges of its tiles of 16 tokens and 8 rows and of the eighths of K."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1, 15, 16, 17, 200])
@pytest.mark.parametrize("E,K", [(1, 32), (8, 224), (9, 256), (16, 2048), (17, 1024), (25, 288), (32, 4096)])
def test_router_logits(T, E, K):
    from llmplayer_b200.kernels import ops
    g = torch.Generator(device=DEV).manual_seed(T + E)
    x = torch.randn(T, K, generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn(E, K, generator=g, device=DEV) * K ** -0.5).to(torch.bfloat16)
    assert ops.router_logits_serves(x, w)
    assert not ops.router_logits_serves(x, w.new_empty(33, K))
    wide = torch.full((T, E + 3), 7.0, device=DEV)
    ops.router_logits(x, w, wide[:, 1:1 + E])
    want = x.double() @ w.double().T
    # float32 sums of K exact products: K / 8 roundings in a chain, of 2^-23 each where the tensor cores cut off
    assert float((wide[:, 1:1 + E].double() - want).norm() / want.norm()) < 2.0 ** -23 * (K / 8 + 8)
    assert float((wide[:, 0] - 7.0).abs().max()) == 0.0 and float((wide[:, 1 + E:] - 7.0).abs().max()) == 0.0
    alone = torch.empty(1, E, device=DEV)
    ops.router_logits(x[T - 1:], w, alone)                # a token's result does not depend on the tokens beside it
    assert torch.equal(alone[0], wide[T - 1, 1:1 + E])
