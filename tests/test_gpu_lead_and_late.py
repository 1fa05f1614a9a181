"""Portions and decoding requests of one step beside each other: the bits of one after the other, with a kernel right in front that writes
queries, keys and values."""
import pytest
import torch

from test_gpu_kernels import err_word

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("hd,nh,kvh,decoding,prompts,window", [(128, 16, 8, 40, [700, 33], 0), (128, 8, 2, 3, [1500], 200), (64, 8, 8, 70, [90, 2, 400], 0),
                                                               (256, 16, 1, 9, [300], 0), (256, 4, 2, 1, [129, 64], 100)])
def test_beside_and_behind(hd, nh, kvh, decoding, prompts, window):
    from vllm_oxide_b200 import kernels
    from vllm_oxide_b200.parts.attention import decode_splits
    from vllm_oxide_b200.parts.base import RotationRule
    bs, width = 64, (nh + 2 * kvh) * hd
    ctx = [1 + 37 * i % 1100 for i in range(decoding)] + prompts
    new = [1] * decoding + prompts
    B, T = len(ctx), sum(new)
    pages = [-(-n // bs) for n in ctx]
    table, at = torch.zeros(B, max(pages), dtype=torch.int32), 0
    for b in range(B):
        table[b, :pages[b]] = torch.arange(at, at + pages[b], dtype=torch.int32)
        at += pages[b]
    pos = [c - n + j for c, n in zip(ctx, new) for j in range(n)]
    req = [b for b, n in enumerate(new) for _ in range(n)]
    slots = i32([int(table[b, p // bs]) * bs + p % bs for b, p in zip(req, pos)])
    cu = [0] + torch.tensor(new).cumsum(0).tolist()
    table, cu_q, ctx_lens, positions = table.to(DEV), i32(cu), i32(ctx), i32(pos)
    g = torch.Generator(device=DEV).manual_seed(hd + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    ang = rnd(1600, hd // 2)
    rule = RotationRule(torch.cat([ang.cos(), ang.sin()], 1).contiguous(), hd, False)
    k0, v0, wn = rnd(at, kvh, bs, hd).bfloat16(), rnd(at, kvh, bs, hd).bfloat16(), rnd(hd)
    splits = decode_splits(B, kvh, max(ctx), kernels.sm_count())
    scratch = torch.empty(max(1, kernels.attention_decode_scratch_floats(hd, B, nh, splits)), device=DEV)
    pairs, err, k, v = kernels.decode_pairs_counter(DEV), err_word(), k0.clone(), v0.clone()
    qkv, out = torch.empty(T, width, dtype=torch.bfloat16, device=DEV), torch.empty(T, nh * hd, dtype=torch.bfloat16, device=DEV)

    def step(rows, beside):
        qkv.copy_(rows)
        kernels.qk_norm_rope_kv_write(qkv, None, positions, slots, wn, wn, rule, k, v, T, nh, kvh, hd, 1e-6, True, err)
        late = kernels.attention_prefill(qkv, width, out, k, v, table, cu_q, ctx_lens, B, max(new), nh, kvh, hd, window, hd ** -0.5, err,
                                         portions=len(prompts), portion_tokens=sum(prompts), lead=beside)
        assert late == beside
        kernels.attention_decode(qkv, width, out, k, v, table, cu_q, ctx_lens, B, nh, kvh, hd, window, hd ** -0.5, splits, scratch, err, pairs=pairs, late=late)
        # a kernel behind both, launched early like every kernel of a step
        kernels.sigmoid_gate_mul(out, qkv[:, :nh * hd], nh * hd)
    steps = [rnd(T, width).bfloat16() for _ in range(4)]
    want = []
    for rows in steps:
        step(rows, False)
        want.append(out.clone())
    got = []
    for _ in range(6):                                  # without a wait between the steps
        for rows in steps:
            step(rows, True)
            got.append(out.clone())
    assert int(err.item()) == 0
    for i, o in enumerate(got):
        assert torch.equal(o, want[i % 4])
