"""The scans with one decay a head and token, 16 tokens at a time on the tensor cores, against the recurrence in 64 bits and
against the walk by multiply-adds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def recurrence(q, k, v, keep, put, state):
    """One head in 64 bits: q, k [T, dk], v [T, dv], keep and put [T], state [dk, dv]; the outputs and the last state."""
    S, out = state.clone(), []
    for i in range(q.shape[0]):
        S = S * keep[i] + put[i] * k[i][:, None] * v[i][None, :]
        out.append(S.T @ q[i])
    return torch.stack(out), S


def error(a, want):
    return ((a.double().cpu() - want).norm() / want.norm()).item()


# dk, dv, heads, tokens of the requests: edges of a chunk, of the 32 columns of a block and of the padded rows
SHAPES = [(128, 128, 2, [1, 2, 15, 16, 17, 1]), (128, 128, 2, [300]), (64, 64, 2, [33, 47, 1]), (96, 40, 3, [31, 1, 5]),
          (16, 8, 2, [50, 1]), (33, 129, 1, [18, 64, 1]), (128, 31, 2, [4, 1])]


@pytest.mark.parametrize("kind", ["lightning", "mlstm"])
@pytest.mark.parametrize("shape", SHAPES)
def test_scan_by_chunks(shape, kind):
    """Few roundings of 32 bits (half an ulp is 6e-8) from the 64-bit recurrence, as the walk by multiply-adds, at every edge of a chunk
    (test_no_further_from_64_bits_than_the_walk compares the two where there are tokens enough to); states of earlier steps are
    carried on, other slots stay."""
    from vllm_oxide_b200 import kernels
    dk, dv, heads, lens = shape
    g = torch.Generator().manual_seed(len(lens) * 1000 + dk)
    rnd = lambda *s: torch.randn(*s, generator=g)
    T, B = sum(lens), len(lens)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32)
    slots = torch.arange(B, 0, -1, dtype=torch.int32)
    extra = 1 if kind == "mlstm" else 0
    state0 = rnd(B + 2, (heads * (dk * (dv + extra) + extra) + 3) // 4 * 4) * 0.3
    if kind == "mlstm":
        state0[:, heads * dk * (dv + 1):] = 0.1
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    dev = lambda t: t.to(DEV)
    rows = rnd(T, heads * (2 * dk + dv) + 2 * heads + heads * dv).bfloat16()
    q, k, v = (x.double().view(T, heads, -1) for x in rows[:, :heads * (2 * dk + dv)].split([heads * dk, heads * dk, heads * dv], 1))
    if kind == "lightning":
        q, k, v = (torch.nn.functional.silu(x) for x in (q, k, v))
        decays = torch.rand(heads, generator=g) * 0.3 + 0.7
        keep, put = decays.double().expand(T, heads), torch.ones(T, heads, dtype=torch.float64)
    else:
        cap, off = 15.0, heads * (2 * dk + dv)
        bi, bf = rnd(heads), rnd(heads) + 3.0
        zi, zf = rows.double()[:, off:off + heads] + bi.double(), rows.double()[:, off + heads:off + 2 * heads] + bf.double()
        li, lf = cap * torch.tanh(zi / cap), -torch.nn.functional.softplus(-cap * torch.tanh(zf / cap))
        keep, put, q = torch.empty(T, heads).double(), torch.empty(T, heads).double(), q * dk ** -0.5
        for b in range(B):
            m = state0[int(slots[b]), heads * dk * (dv + 1):heads * dk * (dv + 1) + heads].double()
            for t in range(int(cu[b]), int(cu[b + 1])):
                new = torch.maximum(lf[t] + m, li[t])
                keep[t], put[t], m = torch.exp(lf[t] + m - new), torch.exp(li[t] - new), new
    got = {}
    for by_chunks in (True, False):
        state, raw, nq = dev(state0), torch.full((T, heads * dv), float("nan"), device=DEV), torch.zeros(T, heads, device=DEV)
        if kind == "lightning":
            kernels.lightning_scan(dev(rows), dev(decays), state, dev(cu), dev(slots), raw, B, heads, dk, dv, err, by_chunks=by_chunks)
        else:
            kernels.mlstm_scan(dev(rows), heads * (2 * dk + dv), heads * (2 * dk + dv) + heads, heads * (2 * dk + dv) + 2 * heads, dev(bi),
                               dev(bf), torch.ones(heads * dv, device=DEV), state, dev(cu), dev(slots), B, heads, dk, dv, dk ** -0.5, cap,
                               1e-6, err, gates=torch.empty(T, heads * 4, device=DEV), raw=raw, nq=nq, by_chunks=by_chunks)
        got[by_chunks] = raw.view(T, heads, dv), state, nq
    assert int(err.item()) == 0
    idle = [s for s in range(B + 2) if s not in slots.tolist()]
    assert torch.equal(got[True][1][idle].cpu(), state0[idle])
    for b in range(B):
        at, slot = slice(int(cu[b]), int(cu[b + 1])), int(slots[b])
        for h in range(heads):
            S0 = state0[slot, h * dk * dv:(h + 1) * dk * dv].double()
            want, S1 = recurrence(q[at, h], k[at, h], v[at, h], keep[at, h], put[at, h], S0.view(dk, dv))
            worst = [error(got[way][0][at, h], want) for way in (True, False)]
            assert worst[0] <= max(3e-7, 1.5 * worst[1]), worst
            ends = [error(got[way][1][slot, h * dk * dv:(h + 1) * dk * dv], S1.reshape(-1)) for way in (True, False)]
            assert ends[0] <= max(3e-7, 1.5 * ends[1]), ends
            if kind == "mlstm":
                n0 = state0[slot, heads * dk * dv + h * dk:heads * dk * dv + (h + 1) * dk].double()[:, None]
                want, n1 = recurrence(q[at, h], k[at, h], torch.ones(T, 1).double()[at], keep[at, h], put[at, h], n0)
                # (a read-out of the normaliser may come near zero: the error counts against the products it is summed of)
                size = (q[at, h].abs().max() * n1.abs().max() * dk ** 0.5).item()
                assert (got[True][2][at, h].double().cpu() - want[:, 0]).abs().max().item() <= 4e-6 * max(size, want.abs().max().item())
                assert error(got[True][1][slot, heads * dk * dv + h * dk:heads * dk * dv + (h + 1) * dk], n1[:, 0]) <= 2e-6


DECAYS = [0.4, 0.493, 0.6, 0.7, 0.8, 0.9, 0.95, 0.98, 0.99, 0.996, 0.999, 1.0]
FORGET_BIAS = [-3.0, -1.0, 0.0, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 8.0]


@pytest.mark.parametrize("dk,dv,T", [(128, 128, 500), (64, 64, 500), (128, 32, 4000)])
@pytest.mark.parametrize("kind", ["lightning", "mlstm"])
def test_no_further_from_64_bits_than_the_walk(kind, dk, dv, T):
    """Head by head, from decays that forget in two tokens to none at all, and over a long text: the read-outs and the state lie no further from
    the recurrence in 64 bits (over the gates that both ways were given) than the walk's.  A tenth and a half of an ulp's tenth are
    what two such errors differ by from draw to draw."""
    from vllm_oxide_b200 import kernels
    heads = len(DECAYS if kind == "lightning" else FORGET_BIAS)
    g = torch.Generator(device=DEV).manual_seed(dk + T)
    W = heads * (2 * dk + dv)
    rows = torch.randn(T, W + 2 * heads + heads * dv, generator=g, device=DEV).bfloat16()
    cu, slots = torch.tensor([0, T], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    n = heads * dk * (dv + 1) + heads
    state0 = torch.randn(1, (n + 3) // 4 * 4, generator=g, device=DEV) * 0.3
    state0[:, heads * dk * (dv + 1):] = 0.1
    err, got = torch.zeros(1, dtype=torch.int32, device=DEV), {}
    gates = torch.empty(T, heads, 4, device=DEV)
    for by_chunks in (True, False):
        state, raw = state0.clone(), torch.empty(T, heads * dv, device=DEV)
        if kind == "lightning":
            kernels.lightning_scan(rows, torch.tensor(DECAYS, device=DEV), state, cu, slots, raw, 1, heads, dk, dv, err, by_chunks=by_chunks)
        else:
            kernels.mlstm_scan(rows, W, W + heads, W + 2 * heads, torch.zeros(heads, device=DEV), torch.tensor(FORGET_BIAS, device=DEV),
                               torch.ones(heads * dv, device=DEV), state, cu, slots, 1, heads, dk, dv, dk ** -0.5, 15.0, 1e-6, err,
                               gates=gates.view(T, heads * 4), raw=raw, nq=torch.empty(T, heads, device=DEV), by_chunks=by_chunks)
        got[by_chunks] = raw.view(T, heads, dv), state[0, :heads * dk * dv].view(heads, dk, dv)
    assert int(err.item()) == 0
    q, k, v = (x.double().view(T, heads, -1) for x in rows[:, :W].split([heads * dk, heads * dk, heads * dv], 1))
    if kind == "lightning":
        q, k, v = (torch.nn.functional.silu(x) for x in (q, k, v))
        keep, put = torch.tensor(DECAYS, device=DEV).double().expand(T, heads), torch.ones(T, heads, device=DEV).double()
    else:
        q = q * float(torch.tensor(dk ** -0.5))
        keep, put = gates[:, :, 0].double(), gates[:, :, 1].double()
    S, want = state0[0, :heads * dk * dv].view(heads, dk, dv).double(), []
    for t in range(T):
        S = torch.baddbmm(S * keep[t][:, None, None], (k[t] * put[t][:, None])[:, :, None], v[t][:, None, :])
        want.append((S.transpose(1, 2) @ q[t][:, :, None])[:, :, 0])
    want = torch.stack(want)
    for h in range(heads):
        for got_here, exact in ((lambda way: got[way][0][:, h], want[:, h]), (lambda way: got[way][1][h], S[h])):
            mine, walk = (((got_here(way).double() - exact).norm() / exact.norm()).item() for way in (True, False))
            assert mine <= 1.1 * walk + 3e-9, (h, mine, walk)


# what is planted, and where: (part of the row, token), or the state; the places are the second request's
ODD = {"infinite v": ("v", 21, float("inf")), "NaN in q": ("q", 40, float("nan")), "infinite k": ("k", 17, float("-inf")),
       "NaN in v, first token": ("v", 0, float("nan")), "large v": ("v", 5, 2.0 ** 100), "large k, last token": ("k", 49, 2.0 ** 90),
       "infinite state": ("state", 0, float("inf")), "large state": ("state", 0, 2.0 ** 70)}


@pytest.mark.parametrize("what", list(ODD))
@pytest.mark.parametrize("kind", ["lightning", "mlstm"])
@pytest.mark.parametrize("dk,dv", [(128, 128), (40, 33)])
def test_values_that_are_not_usual(dk, dv, kind, what):
    """Infinities, NaN and numbers near the end of the range go where the walk takes them and nowhere else: not to another request, head or
    column, nor to an earlier token."""
    from vllm_oxide_b200 import kernels
    place, token, value = ODD[what]
    heads, lens = 2, [20, 50, 33]
    T, B, W = sum(lens), len(lens), heads * (2 * dk + dv)
    g = torch.Generator().manual_seed(dk + token)
    rows = torch.randn(T, W + 2 * heads + heads * dv, generator=g).bfloat16()
    state0 = torch.randn(B, (heads * (dk * (dv + 1) + 1) + 3) // 4 * 4, generator=g) * 0.3
    state0[:, heads * dk * (dv + 1):] = 0.1
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    slots, err = torch.arange(B, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(by_chunks):
        state, raw, nq = state0.to(DEV), torch.zeros(T, heads * dv, device=DEV), torch.zeros(T, heads, device=DEV)
        if kind == "lightning":
            kernels.lightning_scan(rows.to(DEV), torch.tensor([0.9, 0.5], device=DEV), state, cu, slots, raw, B, heads, dk, dv, err,
                                   by_chunks=by_chunks)
        else:
            kernels.mlstm_scan(rows.to(DEV), W, W + heads, W + 2 * heads, torch.zeros(heads, device=DEV), torch.full((heads,), 3.0, device=DEV),
                               torch.ones(heads * dv, device=DEV), state, cu, slots, B, heads, dk, dv, dk ** -0.5, 15.0, 1e-6, err,
                               gates=torch.empty(T, heads * 4, device=DEV), raw=raw, nq=nq, by_chunks=by_chunks)
        return raw.cpu(), state.cpu(), nq.cpu()

    clean = run(True)
    if place == "state":
        state0[1, dk * dv + 3 * dv + 7] = value                      # head 1, row 3, column 7
    else:
        rows[lens[0] + token, {"q": 0, "k": heads * dk, "v": 2 * heads * dk}[place] + 5] = value          # head 0, place 5
    mine, walk = run(True), run(False)
    assert int(err.item()) == 0
    odd = 0
    others = [[t for t in range(T) if not lens[0] <= t < lens[0] + lens[1]], [0, 2], [t for t in range(T) if not lens[0] <= t < lens[0] + lens[1]]]
    for x, want, plain, rest in zip(mine, walk, clean, others):
        assert torch.equal(x[rest], plain[rest])
        for is_odd in (torch.isnan, torch.isposinf, torch.isneginf):
            assert torch.equal(is_odd(x), is_odd(want))
        usual = torch.isfinite(want)
        odd += int((~usual).sum()) + int((want[usual].abs() > 1e9).sum())
        # sums of large numbers cancel: an error counts against the largest of its row and column
        most = torch.where(usual, want, 0.0).abs()
        size = torch.maximum(most.amax(dim=1, keepdim=True), most.amax(dim=0, keepdim=True))[usual]
        assert ((x[usual] - want[usual]).abs() <= 1e-5 * size).all()
    assert odd > 0


def test_which_steps_go_by_chunks():
    """The rule: bfloat16 heads of up to 128 rows whose longest portion is the shorter way on the tensor cores."""
    from vllm_oxide_b200 import kernels
    by = lambda dtype, T, B, longest, dk, exact, heads=16: kernels.matrix_scan_by_chunks(dtype, T, B, longest, heads, dk, 128, exact)
    for exact in (True, False):
        assert not by(torch.bfloat16, 64, 64, 1, 128, exact)              # one token each: nothing to cut
        assert not by(torch.float32, 1525, 25, 1501, 128, exact)
        assert not by(torch.bfloat16, 1525, 25, 1501, 129, exact)
        assert by(torch.bfloat16, 1525, 25, 1501, 128, exact)             # a long portion beside single tokens
        assert by(torch.bfloat16, 3165, 3, 1777, 64, exact)
        assert not by(torch.bfloat16, 2048, 1, 2048, 128, exact)          # one portion: the walk's ranges fill the device
    assert by(torch.bfloat16, 4001, 1, 4001, 128, True, 32) and not by(torch.bfloat16, 4001, 1, 4001, 128, False, 32)


def test_a_slot_out_of_range_is_reported():
    from vllm_oxide_b200 import kernels
    err, one = torch.zeros(1, dtype=torch.int32, device=DEV), torch.ones(1, device=DEV)
    rows = torch.zeros(20, 48, dtype=torch.bfloat16, device=DEV)
    kernels.lightning_scan(rows, one, torch.zeros(2, 256, device=DEV), torch.tensor([0, 20], dtype=torch.int32, device=DEV),
                           torch.tensor([2], dtype=torch.int32, device=DEV), torch.zeros(20, 16, device=DEV), 1, 1, 16, 16, err, by_chunks=True)
    assert int(err.item()) == 4      # VOB_ERR_SLOT


@pytest.mark.parametrize("kind", ["lightning", "mlstm"])
def test_a_layer_beside_decoding_requests_goes_by_chunks(kind, monkeypatch):
    """A portion of 500 tokens beside 24 requests that decode: the layer takes the chunks by the rule, every request goes on from its own
    state, and what follows (decoding, by the walk) finds the states that the chunks left."""
    from helpers import Alone, assert_close, held, rand
    from plain import laruzen_plain, nesezen_plain
    from test_gpu_nesezen_parts import draw, hold, load
    from vllm_oxide_b200 import kernels
    from vllm_oxide_b200.parts import PartSpec, build_part
    dt, D, eps, sizes = torch.bfloat16, 40, 1e-5, dict(num_heads=3, dim=128, vdim=128)
    if kind == "lightning":
        part = build_part("mixer", PartSpec("lightning_attention", dict(hidden_size=D, decay=[0.999, 0.9, 0.5], eps=eps, prefix="m.", **sizes)), dtype=dt,
                          device=DEV)
    else:
        part = build_part("mixer", PartSpec("mlstm", dict(hidden_size=D, gate_cap=6.0, eps=eps, prefix="m.", **sizes)), dtype=dt, device=DEV)
    w = draw(part, 17)
    load(part, w, dt)
    wh, ways = hold(part, w, dt), []
    name = kind + "_scan"
    scan = getattr(kernels, name)
    monkeypatch.setattr(kernels, name, lambda *a, **k: (ways.append(bool(k.get("by_chunks"))), scan(*a, **k))[1])
    alone = Alone([part], dt, block_size=16, pages=80, slots=25)
    xs = {rid: held(rand((506 if rid == 24 else 9, D), 60 + rid), dt) for rid in range(25)}
    got = {rid: [] for rid in xs}
    for step in ([(rid, 0, 6) for rid in range(24)], [(rid, 6, 7) for rid in range(24)] + [(24, 0, 500)], [(rid, 7, 8) for rid in range(24)] + [(24, 500, 501)],
                 [(24, 501, 506)] + [(rid, 8, 9) for rid in range(24)]):
        out, at = alone.step([(rid, xs[rid][a:b]) for rid, a, b in step])[0], 0
        for rid, a, b in step:
            got[rid].append(out[at:at + b - a])
            at += b - a
    assert ways[1] and not ways[2], ways
    m = dict(heads=3, dim=128, vdim=128)
    for rid, x in xs.items():
        if kind == "lightning":
            want = laruzen_plain.lightning(x, wh, "m.", dict(m, decay=[0.999, 0.9, 0.5]), eps, torch.float64)
        else:
            want = nesezen_plain.mlstm(x, wh, "m.", dict(m, gate_cap=6.0), eps, torch.float64, noise=lambda t: held(t, dt))
        assert_close(torch.cat(got[rid]), want, dt, f"{kind}, request {rid}", 0.04)
