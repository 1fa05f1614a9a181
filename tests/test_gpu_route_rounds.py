"""Routing: as many tokens a block, and blocks an SM, as a step's rounds ask for; a token's experts and weights depend on none of it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W,T", [(256, 592), (256, 1776), (256, 1777), (256, 2368), (252, 2371), (256, 3553), (4096, 591), (4096, 595), (4096, 1184), (4096, 1187)])
def test_a_token_in_large_and_small_steps(W, T, dt):
    from vllm_oxide_b200 import kernels
    E, top = 24, 4
    g = torch.Generator(device=DEV).manual_seed(W + T)
    h, w, shared = torch.randn(T, W, generator=g, device=DEV).to(dt), torch.randn(E, W, generator=g, device=DEV), torch.randn(W, generator=g, device=DEV)

    def route(rows):
        n = rows.shape[0]
        ids, weights, gate = torch.full((n, top), -1, dtype=torch.int32, device=DEV), torch.full((n, top), float("nan"), device=DEV), torch.zeros(n, device=DEV)
        kernels.moe_route(rows, w, None, ids, weights, n, top, 1, 1, normalise=True, w_shared=shared, shared_gate=gate)
        return ids, weights, gate
    whole = route(h)
    parts = [route(h[i:i + 100].contiguous()) for i in range(0, T, 100)]
    for a, b in zip(whole, (torch.cat(p) for p in zip(*parts))):
        assert torch.equal(a, b)
    want = (h.double() @ w.double().T).softmax(-1).topk(top).values
    assert (whole[1].double() - want / want.sum(-1, keepdim=True)).abs().max() <= 1e-3      # (sums of W products in float: 4e-5 of scores up to 200)
