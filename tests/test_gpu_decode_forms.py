"""The forms of the decode kernel: one plane for keys and values held once, and three blocks an SM where there are many."""
import math

import pytest
import torch

from test_gpu_kernels import err_word

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


def setup(B, kvh, nh, hd, bs, longest, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    lens = [1 + (longest - 1) * i // max(1, B - 1) for i in range(B)]
    pages = [-(-n // bs) for n in lens]
    table, at = torch.full((B, max(pages)), -1, dtype=torch.int32), 0
    for b in range(B):
        table[b, :pages[b]] = torch.arange(at, at + pages[b], dtype=torch.int32)
        at += pages[b]
    plane = lambda: torch.randn(at, kvh, bs, hd, generator=g, device=DEV).bfloat16()
    return lens, table.to(DEV), plane(), plane(), torch.randn(B, nh * hd, generator=g, device=DEV).bfloat16(), g


def decode(q, k, v, table, lens, kvh, nh, hd, splits, **options):
    from vllm_oxide_b200 import kernels
    B, out, err = len(lens), torch.full_like(q, float("nan")), err_word()
    n = kernels.attention_decode_scratch_floats(hd, B, nh, splits)
    kernels.attention_decode(q, nh * hd, out, k, v, table, i32(list(range(B + 1))), i32(lens), B, nh, kvh, hd, options.pop("window", 0), 1 / math.sqrt(hd),
                             splits, torch.empty(max(1, n), device=DEV), err, **options)
    assert int(err.item()) == 0
    return out


@pytest.mark.parametrize("hd", [192, 256])
@pytest.mark.parametrize("bs,splits,longest", [(16, 1, 65), (64, 2, 700), (256, 4, 1300), (32, 8, 1027), (64, 12, 2000)])
def test_one_plane_held_once(hd, bs, splits, longest):
    """Bit for bit what keys and values in two planes of the same content give, plain and with kept keys and a bias."""
    lens, table, k, _, q, g = setup(9, 1, 16, hd, bs, longest, splits)
    bias = torch.randn(16, 40, generator=g, device=DEV)
    for options in (dict(), dict(window=100), dict(window=70, keep_first=33, dist_bias=bias)):
        assert torch.equal(decode(q, k, k, table, lens, 1, 16, hd, splits, **options), decode(q, k, k.clone(), table, lens, 1, 16, hd, splits, **options))


@pytest.mark.parametrize("B,kvh,group,splits,bs", [(40, 8, 2, 1, 256), (75, 4, 1, 1, 16), (40, 8, 4, 2, 64), (33, 4, 16, 3, 32)])
def test_many_blocks_with_kept_keys_and_a_bias(B, kvh, group, splits, bs):
    """More blocks than two an SM: the bits of a few requests at a time, and the plain kernel's numbers."""
    from vllm_oxide_b200 import kernels
    nh, hd = kvh * group, 128
    lens, table, k, v, q, g = setup(B, kvh, nh, hd, bs, 1500, B)
    options = dict(window=300, keep_first=64, dist_bias=torch.randn(nh, 32, generator=g, device=DEV))
    got = decode(q, k, v, table, lens, kvh, nh, hd, splits, **options)
    few = torch.cat([decode(q[b:b + 3].contiguous(), k, v, table[b:b + 3].contiguous(), lens[b:b + 3], kvh, nh, hd, splits, **options) for b in range(0, B, 3)])
    assert torch.equal(got, few)
    want, err = torch.zeros(B, nh * hd, device=DEV), err_word()
    kernels.paged_attention_generic(q, nh * hd, want, k, v, table, i32(list(range(B))), i32([n - 1 for n in lens]), B, nh, kvh, hd, 300, 1 / math.sqrt(hd), err,
                                    keep_first=64, dist_bias=options["dist_bias"])
    # weights rounded to 8 bits before they meet the values, and the output's own rounding
    assert (got.float() - want).abs().max() <= 2.0 ** -7 * (v.float().abs().max())
