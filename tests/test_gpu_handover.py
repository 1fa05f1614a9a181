"""Portions' attention that leads and decode attention that is late: every form of the decode kernel, and the launches that are refused."""
import ctypes

import pytest
import torch

from test_gpu_kernels import err_word

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


class Step:
    """A step of decoding requests and portions: q, k and v come from kernels right in front, which are launched early too."""

    def __init__(self, hd, nh, kvh, decoding, prompts, longest, window=0, one_plane=False, splits=None, extras=False):
        from vllm_oxide_b200 import kernels
        from vllm_oxide_b200.parts.attention import decode_splits
        from vllm_oxide_b200.parts.base import RotationRule
        self.hd, self.nh, self.kvh, self.window, self.one_plane, self.prompts = hd, nh, kvh, window, one_plane, prompts
        bs, ctx, new = 64, [1 + (longest - 1) * (i + 1) // decoding for i in range(decoding)] + prompts, [1] * decoding + prompts
        self.B, self.T, self.width = len(ctx), sum(new), (nh + 2 * kvh) * hd
        pages = [-(-n // bs) for n in ctx]
        table, at = torch.zeros(self.B, max(pages), dtype=torch.int32), 0
        for b in range(self.B):
            table[b, :pages[b]] = torch.arange(at, at + pages[b], dtype=torch.int32)
            at += pages[b]
        pos = [c - n + j for c, n in zip(ctx, new) for j in range(n)]
        req = [b for b, n in enumerate(new) for _ in range(n)]
        self.slots = i32([int(table[b, p // bs]) * bs + p % bs for b, p in zip(req, pos)])
        self.table, self.cu_q, self.ctx, self.positions = table.to(DEV), i32([0] + torch.tensor(new).cumsum(0).tolist()), i32(ctx), i32(pos)
        self.g = torch.Generator(device=DEV).manual_seed(hd + self.T)
        rnd = lambda *s: torch.randn(*s, generator=self.g, device=DEV)
        ang = rnd(max(ctx) + 1, hd // 2)
        self.rule, self.wn = RotationRule(torch.cat([ang.cos(), ang.sin()], 1).contiguous(), hd, False), rnd(hd)
        self.k = rnd(at, kvh, bs, hd).bfloat16()
        self.v = self.k if one_plane else rnd(at, kvh, bs, hd).bfloat16()
        self.options = dict(keep_first=40, dist_bias=rnd(nh, 32)) if extras else {}
        self.splits = splits or decode_splits(self.B, kvh, max(ctx), kernels.sm_count())
        self.scratch = torch.empty(max(1, kernels.attention_decode_scratch_floats(hd, self.B, nh, self.splits)), device=DEV)
        self.pairs, self.err = kernels.decode_pairs_counter(DEV), err_word()
        self.qkv, self.out = (torch.empty(self.T, w, dtype=torch.bfloat16, device=DEV) for w in (self.width, nh * hd))
        self.rows = [rnd(self.T, self.width).bfloat16() for _ in range(3)]

    def before(self, rows):
        from vllm_oxide_b200 import kernels
        self.qkv.copy_(rows)
        if self.one_plane:      # (the plane stays; the queries are made right in front)
            kernels.sigmoid_gate_mul(self.qkv, rows, self.width)
        else:
            kernels.qk_norm_rope_kv_write(self.qkv, None, self.positions, self.slots, self.wn, self.wn, self.rule, self.k, self.v, self.T, self.nh,
                                          self.kvh, self.hd, 1e-6, True, self.err)

    def portions(self, lead):
        from vllm_oxide_b200 import kernels
        return kernels.attention_prefill(self.qkv, self.width, self.out, self.k, self.v, self.table, self.cu_q, self.ctx, self.B, max(self.prompts), self.nh,
                                         self.kvh, self.hd, self.window, self.hd ** -0.5, self.err, portions=len(self.prompts),
                                         portion_tokens=sum(self.prompts), lead=lead, **self.options)

    def decode(self, late):
        from vllm_oxide_b200 import kernels
        kernels.attention_decode(self.qkv, self.width, self.out, self.k, self.v, self.table, self.cu_q, self.ctx, self.B, self.nh, self.kvh, self.hd,
                                 self.window, self.hd ** -0.5, self.splits, self.scratch, self.err, pairs=self.pairs, late=late, **self.options)

    def run(self, rows, beside):
        from vllm_oxide_b200 import kernels
        self.before(rows)
        late = self.portions(beside)
        assert late == beside
        self.decode(late)
        kernels.sigmoid_gate_mul(self.out, rows[:, :self.nh * self.hd], self.nh * self.hd)      # launched early, reads both kernels' rows


FORMS = [dict(hd=64, nh=4, kvh=2, decoding=5, prompts=[130, 3], longest=900, extras=True, window=200),
         dict(hd=128, nh=16, kvh=8, decoding=4, prompts=[400], longest=700, extras=True, window=150),                    # two blocks an SM at most
         dict(hd=128, nh=16, kvh=8, decoding=45, prompts=[200, 90], longest=700, extras=True, window=150, splits=1),      # more
         dict(hd=128, nh=8, kvh=2, decoding=2, prompts=[260], longest=9000, splits=12),                                   # and the kernel that merges splits
         dict(hd=128, nh=8, kvh=8, decoding=60, prompts=[2500, 1900, 3000], longest=300),                                             # persistent, portions in several rounds
         dict(hd=192, nh=8, kvh=2, decoding=7, prompts=[150], longest=800), dict(hd=192, nh=8, kvh=2, decoding=7, prompts=[150], longest=800, extras=True),
         dict(hd=192, nh=8, kvh=4, decoding=60, prompts=[150], longest=800, extras=True, splits=1),
         dict(hd=192, nh=16, kvh=1, decoding=9, prompts=[70, 300], longest=1500, one_plane=True),
         dict(hd=256, nh=16, kvh=1, decoding=40, prompts=[300], longest=1500, one_plane=True),
         dict(hd=256, nh=16, kvh=1, decoding=160, prompts=[300], longest=200, one_plane=True),
         dict(hd=256, nh=16, kvh=1, decoding=3, prompts=[300], longest=6000, one_plane=True, extras=True, window=900, splits=10),
         dict(hd=256, nh=8, kvh=4, decoding=50, prompts=[900], longest=400)]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f"{k}{v}" for k, v in f.items()).replace(" ", ""))
def test_every_form_beside_and_behind(form):
    """The bits of one kernel after the other, over steps that nothing waits between."""
    s = Step(**form)
    want = []
    for rows in s.rows:
        s.run(rows, False)
        want.append(s.out.clone())
    got = []
    for _ in range(4):
        for rows in s.rows:
            s.run(rows, True)
            got.append(s.out.clone())
    assert int(s.err.item()) == 0 and all(torch.isfinite(w).all() for w in want)
    for i, o in enumerate(got):
        assert torch.equal(o, want[i % len(want)])


def test_late_without_a_lead_is_refused():
    """Never led, led twice over, led on another stream, led while captured: `late` is taken once for a launch that leads on this stream."""
    from vllm_oxide_b200 import kernels
    s = Step(128, 4, 2, 3, [200], 500)
    with torch.cuda.stream(torch.cuda.Stream()):
        s.before(s.rows[0])
        with pytest.raises(kernels.KernelError, match="cannot be late"):
            s.decode(True)
        assert s.portions(True)
        s.decode(True)
        with pytest.raises(kernels.KernelError, match="cannot be late"):
            s.decode(True)
        assert s.portions(True)
        torch.cuda.current_stream().synchronize()
        with torch.cuda.stream(torch.cuda.Stream()), pytest.raises(kernels.KernelError, match="cannot be late"):
            s.decode(True)
        s.decode(True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        led = s.portions(True)
        s.decode(led)
    assert led is False
    graph.replay()
    assert int(s.err.item()) == 0


def test_a_ticket_that_nobody_gives_comes_back_as_an_error_word(monkeypatch):
    """A word that no leading launch writes: the late kernel's waits run out (shortened here), the error word says so and where, and the
    next step on the same context is right."""
    from vllm_oxide_b200 import kernels
    for form in (dict(hd=128, nh=4, kvh=2, decoding=3, prompts=[200], longest=500), dict(hd=128, nh=8, kvh=8, decoding=60, prompts=[200], longest=300)):
        s = Step(**form)
        s.run(s.rows[0], False)
        want, word = s.out.clone(), i32([0])
        s.before(s.rows[0])
        s.portions(False)
        torch.cuda.synchronize()
        kernels.attention_decode_set_wait_limit(s.hd, 50)
        try:
            with monkeypatch.context() as m:
                m.setattr(kernels, "_late_handover", lambda late: (ctypes.c_void_p(word.data_ptr()), ctypes.c_uint(7)))
                s.decode(True)
            torch.cuda.synchronize()
        finally:
            kernels.attention_decode_set_wait_limit(s.hd, 0)
        assert int(s.err.item()) == 0x20 | 0x400
        s.err.zero_()
        s.run(s.rows[0], True)
        assert int(s.err.item()) == 0 and torch.equal(s.out, want)
