"""The delta rule's two instances: many requests of few tokens take the one with fewer registers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("channel_decay", [False, True])
@pytest.mark.parametrize("dim,vdim", [(128, 128), (64, 40), (33, 17), (16, 8), (200, 64)])
def test_a_request_among_many_and_alone(dim, vdim, channel_decay, dt):
    """The same outputs and states, bit for bit, whether a request's tokens come in a step of many short requests or alone; slots of no request
    stay as they are."""
    from vllm_oxide_b200 import kernels
    heads, kvh, lens = 16, 8, [1] * 30 + [2, 0, 17, 33, 1, 3] + [1] * 10
    T, B = sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(dim + vdim)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    na = heads * dim if channel_decay else heads
    qkv, ab, A, bias = rnd(T, 2 * kvh * dim + heads * vdim), rnd(T, heads + na).to(dt), rnd(heads) * 0.3, rnd(na)
    state0, err = rnd(B + 1, heads * dim * vdim), torch.zeros(1, dtype=torch.int32, device=DEV)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()

    def run(first, last, state):
        raw = torch.full((cu[last] - cu[first], heads * vdim), float("nan"), device=DEV)
        kernels.delta_scan(qkv[cu[first]:cu[last]], ab[cu[first]:cu[last]], 0, heads, A, bias, state, i32([c - cu[first] for c in cu[first:last + 1]]),
                           i32(list(range(first, last))), raw, last - first, heads, kvh, dim, vdim, err, channel_decay=channel_decay)
        return raw
    among, alone = state0.clone(), state0.clone()
    raw = run(0, B, among)
    for b in range(B):
        if lens[b]:
            assert torch.equal(raw[cu[b]:cu[b + 1]], run(b, b + 1, alone))
    assert int(err.item()) == 0 and torch.isfinite(raw).all()
    assert torch.equal(among, alone) and torch.equal(among[B], state0[B]) and torch.equal(among[31], state0[31])


@pytest.mark.parametrize("channel_decay", [False, True])
@pytest.mark.parametrize("dim,vdim,lens", [(128, 128, [1, 40, 15, 0, 17, 200]), (64, 40, [33, 16, 2]), (33, 17, [5, 64]), (16, 8, [3, 50]), (8, 3, [47]),
                                           (200, 64, [9, 31])])
def test_portions_longest_first_and_token_by_token(dim, vdim, lens, channel_decay):
    """Portions of unlike lengths in one step give the bits of the same tokens one a step, and the recurrence in 64 bits."""
    from vllm_oxide_b200 import kernels
    heads, kvh, T, B = 4, 2, sum(lens), len(lens)
    g = torch.Generator(device=DEV).manual_seed(dim + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    na = heads * dim if channel_decay else heads
    qkv, ab, A, bias = rnd(T, 2 * kvh * dim + heads * vdim), rnd(T, heads + na), rnd(heads) * 0.3, rnd(na)
    state0, err = rnd(B, heads * dim * vdim), torch.zeros(1, dtype=torch.int32, device=DEV)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()

    def run(tokens, cu_q, slots, state):
        raw = torch.full((len(tokens), heads * vdim), float("nan"), device=DEV)
        kernels.delta_scan(qkv[tokens].contiguous(), ab[tokens].contiguous(), 0, heads, A, bias, state, i32(cu_q), i32(slots), raw, len(slots), heads, kvh, dim,
                           vdim, err, channel_decay=channel_decay)
        return raw
    whole, single = state0.clone(), state0.clone()
    raw, one = run(list(range(T)), cu, list(range(B)), whole), torch.empty(T, heads * vdim, device=DEV)
    for b in range(B):
        for t in range(cu[b], cu[b + 1]):
            one[t] = run([t], [0, 1], [b], single)[0]
    assert int(err.item()) == 0 and torch.equal(raw, one) and torch.equal(whole, single)
    x, a = qkv.double(), ab.double()
    unit = lambda y: y / (y.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k = (unit(x[:, i * kvh * dim:(i + 1) * kvh * dim].view(T, kvh, dim)).repeat_interleave(heads // kvh, 1) for i in (0, 1))
    v = x[:, 2 * kvh * dim:].view(T, heads, vdim)
    decay = torch.exp(-torch.exp(A.double())[:, None] * torch.nn.functional.softplus((a[:, heads:] + bias.double()).view(T, heads, -1)))
    want = torch.empty(T, heads, vdim, dtype=torch.float64, device=DEV)
    for b in range(B):
        S = state0[b].double().view(heads, vdim, dim)
        for t in range(cu[b], cu[b + 1]):
            S = S * decay[t][:, None, :]
            u = torch.sigmoid(a[t, :heads])[:, None] * (v[t] - (S * k[t][:, None]).sum(-1))
            S = S + u[:, :, None] * k[t][:, None]
            want[t] = (S * q[t][:, None]).sum(-1) * dim ** -0.5
        # a token rounds each state element twice; errors decay with the state: a few hundred units of 2^-24 of the largest
        assert (whole[b].double().view(heads, vdim, dim) - S).abs().max() <= 300 * 2.0 ** -24 * max(1.0, S.abs().max().item())
    assert (raw.double().view(T, heads, vdim) - want).abs().max() <= 300 * 2.0 ** -24 * want.abs().max()
