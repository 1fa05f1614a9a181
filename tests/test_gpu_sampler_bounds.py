"""The bound that top-k gathers from: as many of the threads' maxima as tokens are asked for."""
import pytest
import torch

from plain import sampler_plain as S

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("V,pad", [(5, 0), (1023, 1), (1025, 0), (4101, 3), (40000, 0), (40001, 2)])
def test_top_k_around_the_number_of_threads(V, pad):
    """k below, at and above the block's 1,024 threads, rows shorter than the block, rows that do not start on a 16-byte boundary,
    rows of the type's lowest values and of infinities: the plain sampler's tokens, one by one."""
    from vllm_oxide_b200.sampling import Sampler, row_key
    g = torch.Generator().manual_seed(V)
    base = torch.randn(6, V + pad, generator=g)
    base[4, :] = torch.finfo(torch.float32).min
    base[4, V // 2:V // 2 + 2] = 1.0
    base[5, ::2] = float("-inf")
    logits = base.to(DEV)[:, pad // 2:pad // 2 + V]
    top_k = [min(V - 1, k) for k in (1023, 1024, 1025, 2, 2, 2 if V == 5 else 40)]
    top_p = [1.0, 0.9, 1.0, 0.9, 1.0, 0.8]
    s = Sampler(DEV, 6)
    for trial in range(3):
        keys = [row_key(5 + trial, r, r) for r in range(6)]
        got = s.forward(logits, [1.0] * 6, top_k, top_p, keys).cpu().tolist()
        want = [S.sample_row(logits[r].cpu().numpy(), 1.0, top_k[r], top_p[r] if top_p[r] < 1 else None, keys[r]) for r in range(6)]
        assert got == want


@pytest.mark.parametrize("V", [3, 700, 1000, 5000, 40000])
def test_top_k_of_masked_vocabularies(V):
    """Fewer tokens left than top-k asks for, the others at one value (minus infinity, the type's lowest, a large negative number), and k
    around the most that is gathered by the threads' maxima: the plain sampler's tokens, one by one."""
    from vllm_oxide_b200.sampling import Sampler, row_key
    g = torch.Generator().manual_seed(V)
    masks = [float("-inf"), torch.finfo(torch.float32).min, -1e4]
    logits = torch.randn(6, V, generator=g)
    for r in range(6):
        left = torch.randperm(V, generator=g)[:max(1, min(V // 2, (1, 30, 600)[r % 3]))]
        keep = logits[r, left].clone()
        logits[r] = masks[r % 3]
        logits[r, left] = keep
    logits[5] = torch.randn(V, generator=g)
    top_k = [min(V - 1, k) for k in (2, 50, 960, 961, 512, 960)]
    top_p = [1.0, 0.9, 0.8, 1.0, 0.9, 0.95]
    s, temperature = Sampler(DEV, 6), [1.0, 0.7, 1.5, 1.0, 0.7, 1.0]
    for trial in range(3):
        keys = [row_key(9 + trial, r, r) for r in range(6)]
        got = s.forward(logits.to(DEV), temperature, top_k, top_p, keys).cpu().tolist()
        want = [S.sample_row(logits[r].numpy(), temperature[r], top_k[r], top_p[r] if top_p[r] < 1 else None, keys[r]) for r in range(6)]
        assert got == want
