"""Rows longer than what a thread keeps in registers: query and key/value latents over 1,024 elements, unit heads over 256."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
# a value is rounded to its type once (2^-9 of itself in bfloat16, 2^-24 in float32); the sums, roots and quotients before that are float
BOUND = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("q_rank,kv_rank,rot,rotary", [(1024, 1025, 8, 8), (1536, 192, 64, 64), (1025, 1100, 150, 140), (40, 2000, 3, 2)])
@pytest.mark.parametrize("interleaved", [True, False])
def test_latents(q_rank, kv_rank, rot, rotary, interleaved, dt):
    from vllm_oxide_b200 import kernels
    T, pages, bs, width = 5, 2, 4, kv_rank + rot + 5
    g = torch.Generator(device=DEV).manual_seed(q_rank)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    down, wq, wkv = rnd(T, q_rank + kv_rank + rot).to(dt), rnd(q_rank), rnd(kv_rank)
    freq = torch.rand(rotary // 2, generator=g, device=DEV)
    rule = SimpleNamespace(frequencies=freq, amplitude=1.5, rotary_dim=rotary, interleaved=interleaved)
    pos, slots, err = [0, 3, 17, 200, 9], [6, 0, 3, -1, 7], i32([0])
    cq, cache = torch.empty(T, q_rank, dtype=dt, device=DEV), torch.full((pages, 1, bs, width), 7.0, device=DEV).to(dt)
    kernels.latent_prep(down, wq, wkv, rule, i32(pos), i32(slots), cq, cache, T, q_rank, kv_rank, rot, 1e-6, True, err)
    x = down.double()
    norm = lambda v, w: v / (v.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    close = lambda got, want: (got.double() - want).abs().max() <= BOUND[dt] * max(1.0, want.abs().max().item())
    assert int(err.item()) == 0 and close(cq, norm(x[:, :q_rank], wq))
    rows = cache.view(pages * bs, width)
    latent, part = norm(x[:, q_rank:q_rank + kv_rank], wkv), x[:, q_rank + kv_rank:]
    # (the angle position * frequency is a float product: at 17 it is off by 2^-20)
    ang = (i32(pos).float()[:, None] * freq).double()
    c, s = 1.5 * ang.cos(), 1.5 * ang.sin()
    turned = part.clone()
    a, b = (slice(0, rotary, 2), slice(1, rotary, 2)) if interleaved else (slice(0, rotary // 2), slice(rotary // 2, rotary))
    turned[:, a], turned[:, b] = part[:, a] * c - part[:, b] * s, part[:, b] * c + part[:, a] * s
    for t, slot in enumerate(slots):
        if slot >= 0:
            assert close(rows[slot, :kv_rank], latent[t]) and close(rows[slot, kv_rank:kv_rank + rot], turned[t]) and not rows[slot, kv_rank + rot:].any()
    assert all((rows[s] == 7.0).all() for s in range(pages * bs) if s not in slots)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim,vdim,kd_row,vd_row", [(256, 257, 256, 300), (257, 40, 320, 48), (500, 256, 512, 256)])
@pytest.mark.parametrize("unit", [True, False])
def test_unit_heads(dim, vdim, kd_row, vd_row, unit, dt):
    from vllm_oxide_b200 import kernels
    T, nh, kvh, pages, bs = 3, 5, 2, 2, 2
    g = torch.Generator(device=DEV).manual_seed(dim)
    x = torch.randn(T, (nh + kvh) * dim + kvh * vdim, generator=g, device=DEV)
    slots, err = [3, 0, 2], i32([0])
    q = torch.empty(T, nh * kd_row, dtype=dt, device=DEV)
    kc, vc = torch.full((pages, kvh, bs, kd_row), 7.0, device=DEV).to(dt), torch.full((pages, kvh, bs, vd_row), 7.0, device=DEV).to(dt)
    kernels.unit_qk_kv_write(x, i32(slots), q, kc, vc, T, nh, kvh, dim, vdim, 1e-6, unit, True, err)
    heads = x[:, :(nh + kvh) * dim].double().view(T, nh + kvh, dim)
    if unit:
        heads = heads / (heads.square().mean(-1, keepdim=True) + 1e-6).sqrt()
    v = x[:, (nh + kvh) * dim:].double().view(T, kvh, vdim)
    close = lambda got, want: (got.double() - want).abs().max() <= BOUND[dt] * max(1.0, want.abs().max().item())
    q = q.view(T, nh, kd_row)
    assert int(err.item()) == 0 and close(q[:, :, :dim], heads[:, :nh]) and not q[:, :, dim:].any()
    for t, slot in enumerate(slots):
        k_row, v_row = kc[slot // bs, :, slot % bs], vc[slot // bs, :, slot % bs]
        assert close(k_row[:, :dim], heads[t, nh:]) and not k_row[:, dim:].any() and close(v_row[:, :vdim], v[t]) and not v_row[:, vdim:].any()
    assert (kc[0, :, 1] == 7.0).all() and (vc[0, :, 1] == 7.0).all()
