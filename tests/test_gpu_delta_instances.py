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
