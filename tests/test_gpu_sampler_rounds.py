"""Sampler: batches around what clusters of each size hold at once, rows with NaN, short rows with a large k."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def tokens(logits, k, p, first, rows):
    """Tokens of `rows` rows from `first` on, drawn with those rows' settings and keys."""
    from vllm_oxide_b200.sampling import Sampler, row_key
    at = range(first, first + rows)
    s = Sampler(DEV, logits.shape[0])
    return s.forward(logits[first:first + rows], [(0.7, 1.0, 1.3, 0.0)[r % 4] for r in at], [k] * rows, [p] * rows,
                     [row_key(7, r, k) for r in at]).cpu().tolist()


@pytest.mark.parametrize("k,p", [(0, 1.0), (0, 0.9), (1, 1.0), (50, 0.9)])
def test_rows_around_a_round_of_clusters(k, p):
    g = torch.Generator(device=DEV).manual_seed(k)
    x = torch.randn(160, 40000, generator=g, device=DEV) * torch.linspace(0.01, 5.0, 160, device=DEV)[:, None]
    many = tokens(x, k, p, 0, 160)                        # more rows than SMs: a block each
    for rows in (14, 15, 16, 17, 18, 19, 32, 33, 34, 35, 36, 37, 38, 73, 74, 75):
        assert tokens(x, k, p, 0, rows) == many[:rows]


@pytest.mark.parametrize("V", [9001, 32768])
@pytest.mark.parametrize("k,p", [(0, 1.0), (0, 0.9), (50, 0.9), (256, 0.95), (960, 1.0)])
def test_rows_with_nan(V, k, p):
    """One NaN, a few, more than the threads of a block have maxima, a whole part of the row, nothing else: as by one block a row."""
    g = torch.Generator(device=DEV).manual_seed(V)
    x = torch.randn(160, V, generator=g, device=DEV)
    for r, n in enumerate((1, 3, 49, 50, 600, V // 8, V // 2, V)):
        x[2 * r::16, :n] = float("nan")
        x[2 * r + 1::16, torch.randperm(V, generator=g, device=DEV)[:n]] = float("nan")
    many = tokens(x, k, p, 0, 160)
    for first, rows in ((0, 16), (16, 33), (32, 64)):
        assert tokens(x, k, p, first, rows) == many[first:first + rows]


@pytest.mark.parametrize("V", [301, 1000, 1023, 3000])
@pytest.mark.parametrize("k", [299, 600, 960])
def test_a_short_row_with_a_large_k(V, k):
    """Fewer threads with a token than k: nothing outside the k largest is drawn."""
    g = torch.Generator(device=DEV).manual_seed(V + k)
    x = torch.randn(8, V, generator=g, device=DEV).repeat(20, 1)
    got = tokens(x, k, 1.0, 0, 160)
    rank = x.argsort(1, descending=True).argsort(1)
    assert all(int(rank[r, t]) < k for r, t in enumerate(got))
    # one block a row over the same logits in a row that starts off a 16-byte boundary: one token a thread at a time
    wide = torch.zeros(160, V + 1 + (-V - 1) % 4 + 1, device=DEV)
    off = wide[:, 1:1 + V]
    off.copy_(x)
    assert tokens(off, k, 1.0, 0, 160) == got
