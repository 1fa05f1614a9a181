"""Calls of the portion attention for heads of 192 and 256 that the tcgen05 kernel does not take: another kernel answers them."""
import math

import pytest
import torch

from test_gpu_kernels import run_attention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["output", "queries", "query stride"])
@pytest.mark.parametrize("hd", [192, 256])
def test_calls_without_the_alignment_of_the_tcgen05_kernel(hd, what):
    """An output on 16 bytes, queries on 4, rows of queries 4 bytes apart from a multiple of 16: the answers stay
    those of the plain implementation."""
    from vllm_oxide_b200 import kernels
    nh, kvh, bs = 6, 2, 32

    def attention(q, out, kc, vc, bt, cu_q, ctx, T, nh, kvh, hd, window, err, **_):
        dst, stride = out, nh * hd + (2 if what == "query stride" else 0)
        wide = torch.zeros(T * stride + 8, dtype=torch.bfloat16, device=out.device)
        first = 2 if what == "queries" else 0
        rows = wide[first:first + T * stride].view(T, stride)[:, :nh * hd]
        rows.copy_(q.reshape(T, nh * hd))
        if what == "output":
            dst = torch.empty(out.numel() + 16, dtype=out.dtype, device=out.device)[8:8 + out.numel()].view(out.shape)
            assert dst.data_ptr() % 32 == 16
        kernels.attention_prefill(rows, stride, dst, kc, vc, bt, cu_q, ctx, ctx.shape[0], 200, nh, kvh, hd, window, 1.0 / math.sqrt(hd), err)
        if dst is not out:
            out.copy_(dst)
    got, want = run_attention(attention, torch.bfloat16, nh, kvh, hd, bs, 0, [200, 2, 65], [300, 90, 65])
    # (two roundings to bfloat16 of values of order one, as for every case of these kernels)
    assert torch.allclose(got, want, rtol=2e-2, atol=2e-2)


def test_a_scale_of_zero_and_below():
    """With a scale of zero every seen key counts alike; below zero the least product counts most."""
    from vllm_oxide_b200 import kernels
    dev, nh, kvh, hd, n = "cuda:0", 2, 1, 256, 70
    g = torch.Generator(device=dev).manual_seed(7)
    q, k, v = (torch.randn(n if i == 0 else 128, (nh if i == 0 else kvh) * hd, generator=g, device=dev).bfloat16() for i in range(3))
    kc, vc = k.view(2, 64, 1, hd).transpose(1, 2).contiguous(), v.view(2, 64, 1, hd).transpose(1, 2).contiguous()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
    for scale in (0.0, -0.05):
        out, err = torch.empty(n, nh * hd, device=dev, dtype=torch.bfloat16), i32([0])
        kernels.attention_prefill(q, nh * hd, out, kc, vc, i32([[0, 1]]), i32([0, n]), i32([n]), 1, n, nh, kvh, hd, 0, scale, err)
        assert int(err.item()) == 0
        s = torch.einsum("thd,kd->htk", q.double().view(n, nh, hd), k[:n].double()) * scale
        s = s.masked_fill(torch.ones(n, n, device=dev).triu(1).bool(), -math.inf)
        want = torch.einsum("htk,kd->thd", torch.softmax(s, 2), v[:n].double()).reshape(n, -1)
        assert torch.allclose(out.double(), want, rtol=2e-2, atol=2e-2)
