"""Recurrences a channel, two channels a thread and one: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


def shifted(t):
    """The same tensor one element off a boundary of two."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)
    buf[1:] = t.flatten()
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W,lens,chunks", [(2, [1, 9], 8), (30, [7, 8, 65], 8), (32, [0, 33, 300], 32), (66, [257, 1], 32), (256, [1055, 31], 32)])
def test_mingru(W, lens, chunks, dt):
    from vllm_oxide_b200 import kernels
    T, B = sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(W + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    zxg, bz, bx, s0 = rnd(T, 3 * W).to(dt), rnd(W).to(dt), rnd(W).to(dt), rnd(B + 1, W)
    cu, err, got = [0] + torch.tensor(lens).cumsum(0).tolist(), i32([0]), []
    for move in (lambda t: t, shifted):
        state, out = s0.clone(), move(torch.full((T, W), float("nan"), device=DEV).to(dt))
        kernels.mingru_scan(move(zxg), bz, bx, state, i32(cu), i32(list(range(B))), out, B, err, chunks=chunks)
        got.append((out.clone(), state))
    assert int(err.item()) == 0 and torch.isfinite(got[0][0]).all()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W,blocks,lens,chunks", [(4, 2, [1, 9], 8), (36, 3, [7, 66], 8), (32, 1, [33, 0, 300], 32), (64, 4, [257, 1], 64), (256, 2, [1055], 64)])
def test_lru(W, blocks, lens, chunks, dt):
    from vllm_oxide_b200 import kernels
    T, B = sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(W + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    u, gates, y, s0 = rnd(T, W).to(dt), rnd(T, blocks, 2, W // blocks), rnd(T, W + 6).to(dt), rnd(B + 1, W + 5)
    vecs, cu, err, got = [rnd(W) for _ in range(4)], [0] + torch.tensor(lens).cumsum(0).tolist(), i32([0]), []
    for move in (lambda t: t, shifted):
        state, out = s0.clone(), move(torch.full((T, W), float("nan"), device=DEV).to(dt))
        kernels.lru_scan(move(u), move(gates), y, *vecs, state, i32(cu), i32(list(range(B))), out, B, blocks, err, chunks=chunks)
        got.append((out.clone(), state))
    assert int(err.item()) == 0 and torch.isfinite(got[0][0]).all()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
