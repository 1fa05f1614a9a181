"""Many decoding requests of one split: the order in which pairs are given out, and planes that are both keys and values."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


def decode(hd, nh, kvh, ctx, one_plane, pairs, skip=()):
    """Outputs of one step; requests in `skip` bring two tokens and are not this kernel's."""
    from vllm_oxide_b200 import kernels
    from test_gpu_kernels import err_word
    bs, B, new = 64, len(ctx), [2 if b in skip else 1 for b in range(len(ctx))]
    g = torch.Generator(device=DEV).manual_seed(hd + B)
    pages = [-(-n // bs) for n in ctx]
    table, at = torch.zeros(B, max(pages), dtype=torch.int32), 0
    for b in range(B):
        table[b, :pages[b]] = torch.arange(at, at + pages[b], dtype=torch.int32)
        at += pages[b]
    k = torch.randn(at, kvh, bs, hd, generator=g, device=DEV).bfloat16()
    v = k if one_plane else torch.randn(at, kvh, bs, hd, generator=g, device=DEV).bfloat16()
    q = torch.randn(sum(new), nh * hd, generator=g, device=DEV).bfloat16()
    out, err = torch.full_like(q, 7.0), err_word()
    counter = kernels.decode_pairs_counter(DEV) if pairs else None
    kernels.attention_decode(q, nh * hd, out, k, v, table.to(DEV), i32([0] + torch.tensor(new).cumsum(0).tolist()), i32(ctx), B, nh, kvh, hd, 0, hd ** -0.5, 1,
                             None, err, pairs=counter)
    assert int(err.item()) == 0 and (counter is None or not counter.any())
    return out


@pytest.mark.parametrize("lengths", ["one tile", "two tiles", "three tiles", "spread", "one long", "rising"])
@pytest.mark.parametrize("B", [75, 300, 1024, 1025])
def test_order_of_pairs(B, lengths):
    """A block a pair or persistent blocks, in the batch's order or the longest first: the same bits."""
    g = torch.Generator().manual_seed(B)
    draw = lambda lo, hi: torch.randint(lo, hi + 1, (B,), generator=g).tolist()
    ctx = {"one tile": draw(1, 64), "two tiles": draw(1, 128), "three tiles": draw(60, 192), "spread": draw(1, 700), "one long": draw(1, 30),
           "rising": [1 + 2 * b % 500 for b in range(B)]}[lengths]
    if lengths == "one long":
        ctx[B // 2] = 17000          # more tiles than there are buckets
    skip = (3, B - 1) if lengths == "spread" else ()
    for b in skip:
        ctx[b] += 1
    for nh in (4, 16):               # 1 and 4 heads a key head
        assert torch.equal(decode(128, nh, 4, ctx, False, True, skip), decode(128, nh, 4, ctx, False, False, skip))


@pytest.mark.parametrize("hd", [192, 256])
@pytest.mark.parametrize("B", [149, 297, 310])
def test_many_requests_of_one_plane(hd, B):
    """More pairs than persistent blocks fit: a plane that is both keys and values takes a block a pair with and without the counter."""
    g = torch.Generator().manual_seed(B)
    ctx = torch.randint(1, 500, (B,), generator=g).tolist()
    assert torch.equal(decode(hd, 16, 1, ctx, True, True), decode(hd, 16, 1, ctx, True, False))
