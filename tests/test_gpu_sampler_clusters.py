"""Rows shared by the blocks of a cluster: the tokens of a row do not depend on how many blocks it has."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rows_of(V, seed):
    """Rows that take every way through the sampler, flat and peaked, masked in stretches, constant, with infinities and with NaN."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(12, V, generator=g) * torch.linspace(0.01, 6.0, 12)[:, None]
    x[2, : V // 2] = float("-inf")
    x[3, V // 8:] = torch.finfo(torch.float32).min
    x[4, 200:] = -1e4
    x[5] = 1.25
    x[6, ::3] = 2.0
    x[7, V - 1] = 50.0
    x[8, 5] = float("inf")
    x[9] = torch.round(x[9])
    return x


@pytest.mark.parametrize("V,pad", [(4097, 0), (9001, 1), (32768, 0), (32771, 3), (151936, 0)])
@pytest.mark.parametrize("k,p", [(0, 1.0), (0, 0.9), (1, 1.0), (50, 0.9), (20, 1.0), (256, 0.95), (257, 0.9), (960, 0.8), (961, 1.0), (0, 0.1)])
def test_one_row_and_many(V, pad, k, p):
    from vllm_oxide_b200.sampling import Sampler, row_key
    x = rows_of(V, V + k)
    R = x.shape[0]
    wide = torch.zeros(200, V + pad, device=DEV)
    logits = wide[:, pad // 2:pad // 2 + V]
    logits.copy_(x[torch.arange(200) % R].to(DEV))
    s = Sampler(DEV, 200)
    temperature = [(0.7, 1.0, 1.3, 0.0)[r % 4] for r in range(200)]
    keys = [row_key(V, r % R, k) for r in range(200)]
    settings = lambda a, b: (temperature[a:b], [k] * (b - a), [p] * (b - a), keys[a:b])
    many = s.forward(logits, *settings(0, 200)).cpu().tolist()            # more rows than SMs: a block each
    for rows in (1, 12, 24, 48):                                         # eight, eight, four and two blocks a row
        for a in range(0, 12 if rows == 1 else rows, rows):
            assert s.forward(logits[a:a + rows], *settings(a, a + rows)).cpu().tolist() == many[a:a + rows]
