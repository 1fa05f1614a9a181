"""Filters of four taps over portions shorter than a thread's tokens: every block holds several."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dt,to", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("C", [2, 258])
@pytest.mark.parametrize("lens", [[1] * 259, [2] * 150, [3] * 90, [5] * 60, [7, 1, 9] * 17, [15] * 20, [0, 4, 0, 257], [6] * 50 + [0, 0]])
def test_short_portions(lens, C, dt, to):
    """Two channels a thread and one (rows one element off a boundary of two): the same bits.  A portion without a slot gives an error and leaves
    its rows, and padded tokens theirs, as they are; the others' do not change."""
    from vllm_oxide_b200 import kernels
    T, B = sum(lens) + 3, len(lens)
    g = torch.Generator(device=DEV).manual_seed(C + T)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x, w, state, bi, bo = rnd(T, C + 4).to(dt), rnd(C, 4), rnd(B, 1 + 3 * C), rnd(C), rnd(C)
    cu = [0] + torch.tensor(lens).cumsum(0).tolist()
    req = i32([b for b, n in enumerate(lens) for _ in range(n)] + [-1] * 3)

    def run(moved, slots):
        err = i32([0])
        xs, out = x, torch.full((T, C), 7.0, device=DEV).to(to)
        if moved:
            buf = torch.empty(x.numel() + 1, dtype=dt, device=DEV)
            buf[1:] = x.flatten()
            xs = buf[1:].view(x.shape)
        kernels.short_conv_silu(xs, C, w, state, 1, req, i32(cu), i32(slots), out, T, err, bias_in=bi, bias_out=bo)
        return out, int(err.item())
    want, code = run(True, list(range(B)))
    assert code == 0 and torch.isfinite(want).all() and (want[T - 3:] == 7.0).all()
    got, code = run(False, list(range(B)))
    assert code == 0 and torch.equal(got, want)
    lost = next(b for b in range(B // 3, B) if lens[b])
    got, code = run(False, [-1 if b == lost else b for b in range(B)])
    want[cu[lost]:cu[lost + 1]] = 7.0
    assert code != 0 and torch.equal(got, want)
