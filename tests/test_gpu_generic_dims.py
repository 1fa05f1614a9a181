"""The plain attention kernel at every number of value dims a lane may hold, and the float product at the edges of its K slices."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,vd", [(5, 3), (30, 17), (32, 32), (64, 33), (72, 65), (128, 128), (200, 129), (256, 256), (300, 257), (512, 512)])
def test_attention_of_every_size(hd, vd, dt):
    """Ragged contexts through scattered pages, one of which does not exist: its keys are left out and the error word says so."""
    from vllm_oxide_b200 import kernels
    bs, nh, lens = 16, 2, [1, 7, 31, 33, 70]
    g = torch.Generator(device=DEV).manual_seed(hd)
    pages = sum(-(-n // bs) for n in lens)
    k, v = (torch.randn(pages, 1, bs, hd, generator=g, device=DEV).to(dt) for _ in range(2))
    table, perm, at = torch.full((len(lens), 5), -1, dtype=torch.int32), torch.randperm(pages).tolist(), 0
    for b, n in enumerate(lens):
        for p in range(-(-n // bs)):
            table[b, p] = perm[at]
            at += 1
    table[4, 2] = pages + 3                                        # keys 32 .. 47 of the last request
    q = torch.randn(len(lens), nh * hd, generator=g, device=DEV).to(dt)
    out, err = torch.full((len(lens), nh * vd), float("nan"), device=DEV).to(dt), torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kernels.paged_attention_generic(q, nh * hd, out, k, v, table.to(DEV), i32(range(len(lens))), i32([n - 1 for n in lens]), len(lens), nh, 1, hd, 0,
                                    hd ** -0.5, err, value_dim=vd)
    assert int(err.item()) == 8
    for b, n in enumerate(lens):
        keys = [i for i in range(n) if table[b, i // bs] < pages]
        rows = [(int(table[b, i // bs]), i % bs) for i in keys]
        kk, vv = (torch.stack([t[p, 0, r] for p, r in rows]).double() for t in (k, v))
        s = q[b].double().view(nh, hd) @ kk.T * hd ** -0.5
        want = (torch.softmax(s, -1) @ vv[:, :vd]).flatten()
        # a chain of hd products moves a score by hd roundings of the products' sizes, a sum of n weights by n more; bfloat16 rounds the output
        bound = (hd + n + 16) * 2.0 ** -24 * (1 + s.abs().max()) * vv.abs().max() + (2.0 ** -8 * want.abs().max() if dt == torch.bfloat16 else 0)
        assert (out[b].double() - want).abs().max() <= bound


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (3, 65, 15), (64, 64, 16), (65, 63, 17), (303, 80, 192), (6, 331, 33), (130, 5, 80)])
def test_float_product_is_one_chain(M, N, K):
    """One chain of multiply-adds over k in ascending order, whatever slice a k falls into: the bits of a row alone."""
    from vllm_oxide_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a, w = (torch.randn(*s, generator=g, device=DEV) for s in ((M, K), (N, K)))
    out, alone = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    kernels.gemm_f32(a, w, out)
    for m in range(M):
        kernels.gemm_f32(a[m:m + 1], w, alone[m:m + 1])
    assert torch.equal(out, alone)
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert ((out.double() - a.double() @ w.double().T).abs() <= bound).all()
