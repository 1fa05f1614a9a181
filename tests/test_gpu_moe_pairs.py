"""The experts' product on pairs of SMs: row tiles alone and beside a neighbour of the same expert, ragged widths and depths; the logits
of many rows by the same kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rounded(x):
    return x.to(torch.bfloat16).double()


# rows of every expert (0: none), so that tiles of one expert start on even and odd places; widths around a block's 128 and a pair's 256
# rows of W, depths around a stage's 64 columns
@pytest.mark.parametrize("counts", [[1], [128, 129, 1], [256, 0, 130, 257], [5, 300, 640, 0, 3, 128]])
@pytest.mark.parametrize("N,K", [(128, 64), (130, 72), (256, 200), (386, 1032)])
@pytest.mark.parametrize("kind", ["relu2", "float", "pairs", "clamped"])
def test_experts_product(counts, N, K, kind):
    from vllm_oxide_b200 import kernels
    g = torch.Generator().manual_seed(sum(counts) + N)
    E, tile = len(counts), kernels.moe_tc5_row_tile()
    rows, experts, live = [], [], []
    for e, n in enumerate(counts):
        padded = (n + tile - 1) // tile * tile
        live += [True] * n + [False] * (padded - n)
        experts += [e] * (padded // 64)
    total = len(live) + tile                      # a row tile past the end
    experts += [-1] * (tile // 64)
    live += [False] * tile
    a = torch.randn(total, K, generator=g).bfloat16()
    w = (torch.randn(E, N, K, generator=g) / K ** 0.5).bfloat16()
    weight = torch.rand(total, generator=g) + 0.5
    token = torch.where(torch.tensor(live), torch.arange(total), -1).int()
    tile_expert = torch.tensor(experts, dtype=torch.int32)
    gated = kind in ("pairs", "clamped")
    width = N // 2 if gated else N
    c = torch.full((total, width), -7.0, dtype=torch.float32 if kind == "float" else torch.bfloat16)
    out, err = c.to(DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.moe_gemm_tc5(a.to(DEV), w.to(DEV), out, token.to(DEV), tile_expert.to(DEV), kind == "relu2", err, silu_pairs=gated,
                         glu_limit=1.5 if kind == "clamped" else 0.0, row_weight=weight.to(DEV) if kind == "pairs" else None)
    assert int(err.item()) == 0
    got = out.cpu().double()
    for r in range(total):
        if not live[r]:
            assert (got[r] == -7.0).all()         # rows that name no token are left alone
    at = torch.tensor(live)
    e_of = tile_expert.long()[torch.arange(total) // 64].clamp(min=0)
    want = torch.empty(total, N, dtype=torch.float64)
    for e in range(E):
        want[e_of == e] = a[e_of == e].double() @ w[e].double().T
    if kind == "relu2":
        want = want.clamp(min=0) ** 2
    elif gated:
        if kind == "pairs":
            want = want * weight.double()[:, None]
        gate, up = want[:, 0::2], want[:, 1::2]
        if kind == "clamped":
            gate, up = gate.clamp(max=1.5), up.clamp(-1.5, 1.5)
            want = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        else:
            want = torch.nn.functional.silu(gate) * up
    # float sums of up to 1,032 products of order 1 / sqrt(K): 1e-5; one rounding to bfloat16 behind them: 2^-8 of the value
    tol = 2e-5 if kind == "float" else 2 ** -8 * want[at].abs() + 2e-5
    assert ((got[at] - want[at]).abs() <= tol).all()


@pytest.mark.parametrize("M", [1, 64, 129, 256, 257, 700])
@pytest.mark.parametrize("N,K", [(331, 80), (1024, 512)])
def test_logits_of_many_rows(M, N, K):
    """Float logits that are bfloat16 numbers, within one rounding of the 64-bit product; nothing is written past the rows."""
    from vllm_oxide_b200 import kernels
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, K, generator=g).bfloat16(), (torch.randn(N, K, generator=g) / K ** 0.5).bfloat16()
    held, err = torch.full((M + 1, N), -7.0, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.logits_tc5(x.to(DEV), w.to(DEV), held[:M], err)
    assert int(err.item()) == 0 and (held[M] == -7.0).all()
    got, want = held[:M].cpu(), x.double() @ w.double().T
    assert torch.equal(got, got.bfloat16().float())
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 2e-5).all()


def test_which_logits_go_by_this_kernel():
    """The rule: wide matrices and rounds of items that leave many SMs idle are the library's, small or full ones this kernel's."""
    from vllm_oxide_b200 import kernels
    pays = lambda rows, vocab, width: kernels.logits_tc5_pays(torch.empty(rows, width, dtype=torch.bfloat16, device=DEV),
                                                              torch.empty(vocab, width, dtype=torch.bfloat16, device=DEV))
    assert pays(1357, 32768, 2048) and pays(512, 32768, 2048) and pays(256, 32768, 4096) and pays(1024, 4096, 1024)
    assert not pays(256, 4096, 2048) and not pays(384, 32768, 4096) and not pays(1024, 32768, 8192)
    assert not pays(512, 32768, 2044)             # a width that is no multiple of 8


@pytest.mark.parametrize("kind,N,K,tiles", [("float", 8200, 72, [6, 5, 5]), ("relu2", 4096, 136, [16, 1, 17]), ("pairs", 2048, 2048, [25, 24, 23]),
                                            ("float", 300, 64, [200, 201]), ("pairs", 520, 64, [300])])
def test_items_of_two_tiles_and_of_one(kind, N, K, tiles):
    """Steps with so many items that two tiles of an expert share one (the last: too little to multiply, so none do): the 64-bit products,
    and rows that name no token left alone."""
    from vllm_oxide_b200 import kernels
    E, rows = len(tiles), 128 * (sum(tiles) + 2)
    g = torch.Generator(device=DEV).manual_seed(N)
    a = torch.randn(rows, K, generator=g, device=DEV).bfloat16()
    w = (torch.randn(E, N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    owner = torch.cat([torch.full((128 * n,), e) for e, n in enumerate(tiles)] + [torch.full((256,), -1)]).int().to(DEV)
    token = torch.where((owner >= 0) & (torch.rand(rows, generator=g, device=DEV) < 0.9), torch.arange(rows, device=DEV).int(), -1)
    gated = kind == "pairs"
    out = torch.full((rows, N // 2 if gated else N), -7.0, dtype=torch.float32 if kind == "float" else torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.moe_gemm_tc5(a, w, out, token, owner[::64].contiguous(), kind == "relu2", err, silu_pairs=gated)
    assert int(err.item()) == 0 and (out[token < 0] == -7.0).all()
    for e in range(E):
        at = (owner == e) & (token >= 0)
        want = a[at].double() @ w[e].double().T
        if kind == "relu2":
            want = want.clamp(min=0) ** 2
        elif gated:
            want = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        # float sums of up to 2,048 products of order 1 / sqrt(K): 2e-5; one rounding to bfloat16 behind them: 2^-8 of the value
        tol = 2e-5 if kind == "float" else 2 ** -8 * want.abs() + 2e-5
        assert ((out[at].double() - want).abs() <= tol).all()
