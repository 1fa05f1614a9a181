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


@pytest.mark.parametrize("dt,to", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("C,lens", [(2, [300]), (34, [1, 9, 250, 0, 40]), (258, [3, 261]), (256, [8] * 33), (512, [257, 1, 2])])
@pytest.mark.parametrize("biases", [False, True])
def test_four_taps(C, lens, dt, to, biases):
    """Portions that begin and end inside a thread's tokens, inputs from the slot, a padded token."""
    from vllm_oxide_b200 import kernels
    T, B = sum(lens) + 1, len(lens)
    g = torch.Generator(device=DEV).manual_seed(C + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, w, state = rnd(T, C + 6).to(dt), rnd(C, 4), rnd(B, 5 + 3 * C)
    bi, bo = (rnd(C), rnd(C)) if biases else (None, None)
    cu, err, got = [0] + torch.tensor(lens).cumsum(0).tolist(), i32([0]), []
    req = i32([b for b, n in enumerate(lens) for _ in range(n)] + [-1])
    for move in (lambda t: t, shifted):
        out = move(torch.full((T, C), 7.0, device=DEV).to(to))
        kernels.short_conv_silu(move(x), C, w, state, 5, req, i32(cu), i32(list(range(B))), out, T, err, activation=not biases, bias_in=bi, bias_out=bo)
        got.append(out.clone())
    assert int(err.item()) == 0 and torch.equal(got[0], got[1]) and (got[0][T - 1] == 7.0).all()
    for b, n in enumerate(lens):
        add = bi.double() if biases else 0.0
        seq = torch.cat([state[b, 5:].double().view(3, C), x[cu[b]:cu[b] + n, :C].double() + add])
        want = sum(seq[k:k + n] * w[:, k].double() for k in range(4)) + (bo.double() if biases else 0.0)
        want = want if biases else want * torch.sigmoid(want)
        if n:       # five roundings of sums of a few units; bfloat16 rounds the output
            assert (got[0][cu[b]:cu[b] + n].double() - want).abs().max() <= 64 * 2.0 ** -24 * 8 + (2.0 ** -8 * want.abs().max() if to == torch.bfloat16 else 0)
