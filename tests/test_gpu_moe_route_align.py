"""Routing for every number of tokens a block, and the sorting of pairs by expert."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,W,E,top", [(1, 8, 1, 1), (5, 30, 3, 2), (147, 132, 17, 4), (297, 260, 16, 4), (593, 128, 7, 3), (1201, 2048, 16, 4), (1190, 3072, 5, 2)])
def test_logits_do_not_depend_on_the_tokens_beside(T, W, E, top, dt):
    """A token's choice and weights, bit for bit, alone and in a block of any size; the softmax over the logits in 64 bits."""
    from vllm_oxide_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(T + W)
    h = torch.randn(T, W, generator=g, device=DEV).to(dt)
    w, bias, ws = (torch.randn(*s, generator=g, device=DEV) / W ** 0.5 for s in ((E, W), (E,), (W,)))

    def route(x):
        n = x.shape[0]
        ids, weights = torch.full((n * top,), -1, dtype=torch.int32, device=DEV), torch.full((n * top,), float("nan"), device=DEV)
        sg = torch.full((n,), float("nan"), device=DEV)
        kernels.moe_route(x, w, None, ids, weights, n, top, 1, 1, router_bias=bias, w_shared=ws, shared_gate=sg)
        return ids.view(n, top), weights.view(n, top), sg
    ids, weights, sg = route(h)
    for t in list(range(0, T, max(1, T // 13))) + [T - 1]:
        one = route(h[t:t + 1].clone())
        assert torch.equal(ids[t], one[0][0]) and torch.equal(weights[t], one[1][0]) and torch.equal(sg[t], one[2][0])
    z = h.double() @ w.double().T + bias.double()
    # a logit is at most W roundings of its products' sizes away
    off = (W + 4) * 2.0 ** -24 * ((h.double().abs() @ w.double().abs().T).max() + 1)
    p = torch.softmax(z, -1)
    assert (weights.double() - p.gather(1, ids.long())).abs().max() <= 4 * off + 1e-6
    assert (z.gather(1, ids.long()) >= torch.topk(z, top).values - 2 * off).all()
    assert (sg.double() - torch.sigmoid(h.double() @ ws.double())).abs().max() <= off + 1e-6


@pytest.mark.parametrize("n,top,E,pad", [(1, 1, 1, 64), (33, 3, 5, 64), (160, 4, 16, 128), (1024, 2, 256, 128), (1032, 4, 257, 64), (16004, 4, 16, 128), (5000, 5, 31, 128)])
def test_pairs_sorted_by_expert(n, top, E, pad):
    """Every pair has a row of its own in its expert's range, ranges are padded, padding names no token; a pair of no expert has no row."""
    from vllm_oxide_b200 import kernels
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, E, (n,), generator=g, dtype=torch.int32)
    ids[torch.rand(n, generator=g) < 0.3] = E // 2                 # one expert has most of them
    if n > 40:
        ids[7], ids[n - 1] = E, -3                                 # no experts
    weights = torch.rand(n, generator=g)
    rows = (n + min(E, n) * (pad - 1) + pad - 1) // pad * pad
    dev = lambda x, m: torch.full((m,), x, dtype=torch.int32, device=DEV)
    slot_of, row_token, tile_expert, row_weight = dev(99, n), dev(99, rows), dev(99, rows // 64), torch.full((rows,), float("nan"), device=DEV)
    kernels.moe_align(ids.to(DEV), slot_of, row_token, tile_expert, n, top, E, pad=pad, weights=weights.to(DEV), row_weight=row_weight)
    slot_of, row_token, tile_expert, row_weight = (t.cpu() for t in (slot_of, row_token, tile_expert, row_weight))
    live = (ids >= 0) & (ids < E)
    counts = torch.bincount(ids[live].long(), minlength=E)
    first = torch.cat([torch.zeros(1, dtype=torch.long), ((counts + pad - 1) // pad * pad).cumsum(0)])
    assert (slot_of[~live] == -1).all() and slot_of[live].unique().numel() == int(live.sum())
    at, e = slot_of[live].long(), ids[live].long()
    assert ((at >= first[e]) & (at < first[e] + counts[e])).all()
    assert torch.equal(row_token[at], (torch.arange(n)[live] // top).int()) and torch.equal(row_weight[at], weights[live])
    assert int((row_token >= 0).sum()) == int(live.sum()) and (row_token >= -1).all()
    want = torch.full((rows // 64,), -1, dtype=torch.int32)
    for x in range(E):
        want[first[x] // 64:first[x + 1] // 64] = x
    assert torch.equal(tile_expert, want)
