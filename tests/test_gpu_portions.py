"""Portions among many decoding requests: which blocks of the attention kernel for portions find work."""
import pytest
import torch

from test_gpu_kernels import run_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("known", [True, False])
@pytest.mark.parametrize("query_tiles", [1, 2])
@pytest.mark.parametrize("q_lens", [[1] * 31 + [2], [1] * 32 + [300, 1, 129] + [1] * 70 + [64], [0, 257, 1, 0, 1, 128] + [1] * 40 + [2, 0]],
                         ids=["last lane", "across warps", "empty requests"])
def test_portions_among_decoding_requests(q_lens, query_tiles, known):
    """The blocks are numbered over the portions alone: every portion's rows are written, wherever its request stands (edges of
    the 32 requests a warp looks at, requests without tokens), with the counts known to the host or not."""
    import math
    from vllm_oxide_b200 import kernels
    nh, kvh, hd = 8, 2, 64

    def attention(q, out, kc, vc, bt, cu_q, ctx, T, nh, kvh, hd, window, err, **_):
        lens = (cu_q[1:] - cu_q[:-1]).tolist()
        more = [n for n in lens if n > 1]
        kw = dict(portions=len(more), portion_tokens=sum(more)) if known else {}
        kernels.attention_prefill(q.reshape(T, nh * hd), nh * hd, out, kc, vc, bt, cu_q, ctx, len(lens), max(lens), nh, kvh, hd, window,
                                  1.0 / math.sqrt(hd), err, query_tiles=query_tiles, **kw)
    got, want = run_attention(attention, torch.bfloat16, nh, kvh, hd, 32, 0, q_lens, [n + 37 for n in q_lens])
    at = 0
    for n in q_lens:
        if n > 1:
            # (two roundings to bfloat16 of values of order one, as for every case of this kernel)
            assert torch.allclose(got[at:at + n], want[at:at + n], rtol=2e-2, atol=2e-2)
        at += n


@pytest.mark.parametrize("hd,block_size,window,nh", [(192, 64, 0, 6), (256, 64, 0, 16), (256, 16, 100, 4), (192, 32, 33, 3), (256, 256, 70, 2)])
def test_keys_and_values_of_one_plane(hd, block_size, window, nh):
    """Heads of 192 and 256 whose keys are their values (a latent): the tcgen05 kernel keeps a stage's rows once."""
    import math
    from vllm_oxide_b200 import kernels

    def same_rows(q, ks, vs, kc, vc, bt, positions):
        vc.copy_(kc)
        for k, v in zip(ks, vs):
            v.copy_(k)

    def attention(q, out, kc, vc, bt, cu_q, ctx, T, nh, kvh, hd, window, err, **_):
        kernels.attention_prefill(q.reshape(T, nh * hd), nh * hd, out, kc, kc, bt, cu_q, ctx, ctx.shape[0], 300, nh, kvh, hd, window,
                                  1.0 / math.sqrt(hd), err)
    got, want = run_attention(attention, torch.bfloat16, nh, 1, hd, block_size, window, [2, 300, 129, 64], [2, 517, 129, 200], craft=same_rows)
    # (two roundings to bfloat16 of values of order one, as for every case of this kernel)
    assert torch.allclose(got, want, rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("kernel", [dict(), dict(use_tc5=False), dict(use_tc5=False, use_tma=False)], ids=["tcgen05", "TMA", "cp.async"])
@pytest.mark.parametrize("hd,bias", [(64, False), (128, True), (192, False), (256, True)])
def test_capped_scores_in_tiles_without_a_mask(hd, bias, kernel):
    """A cap on the scores (and a bias behind it) counts in every tile, also in those that lie wholly before the queries: against
    64 bits, over contexts of many tiles, with scores that the cap changes by half."""
    import math
    from vllm_oxide_b200 import kernels
    dev, nh, kvh, bs, cap = "cuda:0", 4, 2, 64, 4.0
    q_lens, ctx_lens = [70, 2], [700, 300]
    g = torch.Generator(device=dev).manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)
    pages = [-(-c // bs) for c in ctx_lens]
    kc, vc = rnd(sum(pages), kvh, bs, hd).bfloat16(), rnd(sum(pages), kvh, bs, hd).bfloat16()
    bt = torch.full((2, max(pages)), -1, dtype=torch.int32)
    bt[0, :pages[0]], bt[1, :pages[1]] = torch.arange(pages[0]).int(), torch.arange(pages[0], sum(pages)).int()
    T = sum(q_lens)
    q, table = (rnd(T, nh * hd) * 3).bfloat16(), rnd(nh, 400) if bias else None
    cu, ctx = (torch.tensor(x, dtype=torch.int32, device=dev) for x in ([0, q_lens[0], T], ctx_lens))
    out, err, scale = torch.empty(T, nh * hd, device=dev), torch.zeros(1, dtype=torch.int32, device=dev), 1 / math.sqrt(hd)
    kernels.attention_prefill(q, nh * hd, out, kc, vc, bt.to(dev), cu, ctx, 2, max(q_lens), nh, kvh, hd, 0, scale, err, softcap=cap,
                              dist_bias=table, **kernel)
    assert int(err.item()) == 0
    at = 0
    for b, (n, c) in enumerate(zip(q_lens, ctx_lens)):
        rows = bt[b, :pages[b]].long().to(dev)
        k, v = (x[rows].double().transpose(0, 1).reshape(kvh, -1, hd)[:, :c].repeat_interleave(nh // kvh, 0) for x in (kc, vc))
        s = cap * torch.tanh(q[at:at + n].double().view(n, nh, hd).transpose(0, 1) @ k.transpose(1, 2) * scale / cap)
        dist = torch.arange(c - n, c, device=dev)[:, None] - torch.arange(c, device=dev)[None]
        if bias:
            s = s + table.double()[:, dist.clamp(0, table.shape[1] - 1)]
        want = (torch.softmax(s.masked_fill(dist < 0, -math.inf), 2) @ v).transpose(0, 1).reshape(n, -1)
        # probabilities in bfloat16, half an ulp of which is 2^-9: the norm of the error stays below that
        assert ((out[at:at + n].double() - want).norm() / want.norm()).item() < 2 ** -9
        at += n


@pytest.mark.parametrize("hd,nh,kvh,window,one_plane", [(256, 16, 1, 0, True), (256, 8, 4, 300, False), (192, 12, 3, 0, False), (192, 16, 1, 100, True)])
def test_large_heads_are_no_further_from_64_bits(hd, nh, kvh, window, one_plane):
    """The probabilities of a row are rounded to bfloat16 against the row's own maximum, as in the mma.sync kernel, so that the largest is
    exact: the tcgen05 kernel's error against 64 bits is that kernel's (float output, so that nothing hides it)."""
    import math
    from vllm_oxide_b200 import kernels
    dev, bs, n, c = "cuda:0", 64, 300, 1100
    g = torch.Generator(device=dev).manual_seed(hd + nh)
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)
    pages = -(-c // bs)
    kc = rnd(pages, kvh, bs, hd).bfloat16()
    vc = kc if one_plane else rnd(pages, kvh, bs, hd).bfloat16()
    q, scale = (rnd(n, nh * hd) * 1.5).bfloat16(), 1 / math.sqrt(hd)
    bt, err = torch.arange(pages, dtype=torch.int32, device=dev)[None], torch.zeros(1, dtype=torch.int32, device=dev)
    cu, ctx = torch.tensor([0, n], dtype=torch.int32, device=dev), torch.tensor([c], dtype=torch.int32, device=dev)
    k, v = (x.double().transpose(0, 1).reshape(kvh, -1, hd)[:, :c].repeat_interleave(nh // kvh, 0) for x in (kc, vc))
    dist = torch.arange(c - n, c, device=dev)[:, None] - torch.arange(c, device=dev)[None]
    seen = (dist >= 0) & ((dist < window) if window else (dist >= 0))
    s = (q.double().view(n, nh, hd).transpose(0, 1) @ k.transpose(1, 2) * scale).masked_fill(~seen, -math.inf)
    want = (torch.softmax(s, 2) @ v).transpose(0, 1).reshape(n, -1)
    errors = []
    for kernel in (dict(), dict(use_tc5=False)):
        out = torch.empty(n, nh * hd, device=dev)
        kernels.attention_prefill(q, nh * hd, out, kc, vc, bt, cu, ctx, 1, n, nh, kvh, hd, window, scale, err, **kernel)
        assert int(err.item()) == 0
        errors.append(((out.double() - want).norm() / want.norm()).item())
    # (a hundredth: what two sums of the same rounded terms in another order may differ by is far below that)
    assert errors[0] <= 1.01 * errors[1], errors
