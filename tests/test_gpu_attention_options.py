"""The attention kernels for portions and for decoding requests with what a layer may add to the softmax, over random batches, every
head size that is a multiple of 64 and every way to split the keys."""
import math
import random

import numpy as np
import pytest
import torch

from test_gpu_kernels import err_word

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

PORTIONS = {"tcgen05": dict(), "tcgen05, one query tile": dict(query_tiles=1), "tcgen05, rows": dict(tiles_by_tma=False),
            "mma.sync, TMA": dict(use_tc5=False), "mma.sync, cp.async": dict(use_tc5=False, use_tma=False)}


@pytest.mark.parametrize("hd", [64, 128, 192, 256])
@pytest.mark.parametrize("seed", range(8))
def test_random_batches_with_options(hd, seed):
    """Windows with kept first keys, biases by distance, caps, sinks, gates and keys that are their own values, alone and together;
    contexts of up to 47 tiles, so that the kept keys' seam falls inside any split; splits that merge as a cluster (2 to 8) and through
    memory.  Against the plain kernel; each kernel writes its own rows only."""
    from vllm_oxide_b200 import kernels
    rng = random.Random(100 * hd + seed)
    kvh = rng.choice([1, 2, 3, 4])
    nh = kvh * rng.choice([1, 2, 3, 5, 8, 16])
    bs, B = rng.choice([16, 32, 64, 128, 256]), rng.randint(2, 6)
    ctx_lens = [rng.choice([rng.randint(1, 70), rng.randint(1, 700), rng.randint(700, 3000)]) for _ in range(B)]
    q_lens = [1 if (k := rng.random()) < 0.4 else (c if k < 0.6 else rng.randint(1, min(c, 400))) for c in ctx_lens]
    q_lens[0], ctx_lens[1], q_lens[1] = 1, max(ctx_lens[1], 150), 150
    window = rng.choice([0, rng.randint(1, 60), rng.randint(60, 900)])
    keep = rng.choice([0, rng.randint(1, 20), rng.randint(20, 300)]) if window else 0
    g = torch.Generator(device=DEV).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    bias = rnd(nh, rng.choice([3, 200, 4000])) if rng.random() < 0.5 else None
    options = dict(softcap=rng.choice([0.0, 5.0, 30.0]), sink=rng.choice([False, True, rnd(nh)]), keep_first=keep, dist_bias=bias)
    pages = [-(-c // bs) for c in ctx_lens]
    total, T = sum(pages) + 2, sum(q_lens)
    order = torch.randperm(total - 1, generator=torch.Generator().manual_seed(seed)) + 1
    kc = rnd(total, kvh, bs, hd).bfloat16()
    vc = kc if rng.random() < 0.4 else rnd(total, kvh, bs, hd).bfloat16()
    bt, at = torch.full((B, max(pages)), -1, dtype=torch.int32), 0
    for b in range(B):
        bt[b, :pages[b]] = order[at:at + pages[b]].int()
        at += pages[b]
    bt, q = bt.to(DEV), (rnd(T, nh * hd) * rng.choice([0.3, 1.0, 3.0])).bfloat16()
    if rng.random() < 0.5:
        options.update(gate=rnd(T, nh).bfloat16(), gate_stride=nh)
    cu = [0] + [int(x) for x in np.cumsum(q_lens)]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    cu_q, ctx = i32(cu), i32(ctx_lens)
    token_req = i32([b for b, n in enumerate(q_lens) for _ in range(n)])
    positions = i32([c - n + i for n, c in zip(q_lens, ctx_lens) for i in range(n)])
    scale, err = 1.0 / math.sqrt(hd), err_word()
    want = torch.zeros(T, nh * hd, device=DEV)
    kernels.paged_attention_generic(q, nh * hd, want, kc, vc, bt, token_req, positions, T, nh, kvh, hd, window, scale, err, **options)
    single = torch.tensor([cu[b] for b in range(B) if q_lens[b] == 1], dtype=torch.long, device=DEV)
    portion = torch.tensor([t for b in range(B) if q_lens[b] > 1 for t in range(cu[b], cu[b + 1])], dtype=torch.long, device=DEV)
    runs = [(name, portion, single, lambda out, kw=kw: kernels.attention_prefill(
        q, nh * hd, out, kc, vc, bt, cu_q, ctx, B, max(q_lens), nh, kvh, hd, window, scale, err, **options, **kw)) for name, kw in PORTIONS.items()]
    for splits in (1, 2, 3, rng.randint(4, 8), 9, rng.randint(10, 20)):
        n = kernels.attention_decode_scratch_floats(hd, B, nh, splits)
        scratch = torch.empty(max(n, 1), device=DEV) if n else None
        for tma in (True, False):
            runs.append((f"decode, {splits} splits, TMA {tma}", single, portion, lambda out, s=splits, sc=scratch, tma=tma: kernels.attention_decode(
                q, nh * hd, out, kc, vc, bt, cu_q, ctx, B, nh, kvh, hd, window, scale, s, sc, err, use_tma=tma, **options)))
    what = f"nh={nh} kvh={kvh} page={bs} window={window} keep={keep} q={q_lens} ctx={ctx_lens} {sorted(k for k, v in options.items() if v is not None)}"
    for name, mine, others, launch in runs:
        out = torch.full((T, nh * hd), 777.0, device=DEV)
        launch(out)
        assert err.item() == 0, (name, what)
        # (probabilities in bfloat16 beside float ones: 2^-9 of values that reach 5)
        assert (out[mine] - want[mine]).abs().max() < 2e-2, (name, what)
        assert (out[others] == 777).all(), (name, what)


@pytest.mark.parametrize("splits", [1, 2, 5, 8, 11])
@pytest.mark.parametrize("hd,bs", [(64, 64), (128, 16), (256, 256)])
def test_decode_reads_the_right_kept_key(hd, bs, splits):
    """One key decides the output: the last kept one and the window's first are seen in whatever split they fall, their neighbours are not."""
    from vllm_oxide_b200 import kernels
    nh, kvh, ctx, window, keep = 4, 2, 2000, 600, 70
    pages = -(-ctx // bs)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    n = kernels.attention_decode_scratch_floats(hd, 1, nh, splits)
    for key, seen in ((0, True), (keep - 1, True), (keep, False), (ctx - window - 1, False), (ctx - window, True), (ctx - 1, True)):
        kc = torch.zeros(pages, kvh, bs, hd, dtype=torch.bfloat16, device=DEV)
        vc, err = kc.clone(), err_word()
        kc[key // bs, :, key % bs] = 4.0
        vc[key // bs, :, key % bs] = 5.0
        out = torch.empty(1, nh * hd, device=DEV)
        kernels.attention_decode(torch.ones(1, nh * hd, dtype=torch.bfloat16, device=DEV), nh * hd, out, kc, vc,
                                 torch.arange(pages, dtype=torch.int32, device=DEV)[None], i32([0, 1]), i32([ctx]), 1, nh, kvh, hd, window,
                                 1 / math.sqrt(hd), splits, torch.empty(max(n, 1), device=DEV) if n else None, err, keep_first=keep,
                                 dist_bias=torch.zeros(nh, 8, device=DEV))
        assert err.item() == 0
        assert (out > 4.9).all() if seen else (out == 0).all(), (key, out)
