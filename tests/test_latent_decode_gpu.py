"""Latent attention of single tokens over the streamed cache rows against plain sums in 64 bits: lists of tiles that end inside,
at and one past a tile and a page, one CTA's range inside a list and across several, more heads than a tile of rows holds,
windows, rows that pad a captured step, and a far key that stands out."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rank,rot", [(64, 32), (112, 16), (256, 32), (256, 96), (512, 64)])
@pytest.mark.parametrize("heads,lens,window", [(16, [3000, 1, 32, 33, 64, 65, 700], None), (1, [20], None), (9, [5000], None),
                                               (40, [31, 2048, 97], None), (32, [200] * 70, None), (17, [900, 150, 64], 100),
                                               (5, [1] * 300, None)])
def test_single_tokens_over_streamed_rows(rank, rot, heads, lens, window):
    from gemmars_b200 import kernels as k
    torch.manual_seed(rank + heads)
    n, page, kd = len(lens), 64, rank + rot
    width = -(-max(lens) // page)
    pages = sum(-(-m // page) for m in lens)
    cache = torch.randn(pages + 1, page, kd, device=DEV).bfloat16()
    order = (torch.randperm(pages) + 1).tolist()
    table = torch.zeros(n + 1, width, dtype=torch.int32)
    slots = list(range(n))[::-1]
    for i, m in enumerate(lens):
        for j in range(-(-m // page)):
            table[slots[i], j] = order.pop()
    table = table.to(DEV)
    q = (torch.randn(n, heads * kd, device=DEV) * 2 * kd ** -0.5).bfloat16()
    rows = []
    for i, m in enumerate(lens):
        pos = torch.arange(m, device=DEV)
        rows.append(cache[table[slots[i]][pos // page].long(), pos % page].double())
    far = 0 if window is None else max(0, lens[0] - window)
    q[0, :kd] = (rows[0][far] * (8.0 / kd ** 0.5)).bfloat16()          # head 0 of the first sequence points at its first key
    start = torch.tensor([m - 1 for m in lens], dtype=torch.int32, device=DEV)
    slot = torch.tensor(slots, dtype=torch.int32, device=DEV)
    out = torch.zeros(n, heads * rank, device=DEV, dtype=torch.bfloat16)
    k.latent_decode(q, out, heads, rank, rot, cache, table, page, start, slot, window)
    k.check_status()
    again = torch.zeros_like(out)
    k.latent_decode(q, again, heads, rank, rot, cache, table, page, start, slot, window)
    assert torch.equal(out, again)
    for i in sorted({0, 1 % n, 2 % n, n // 2, n - 1}):
        seen = rows[i] if window is None else rows[i][max(0, lens[i] - window):]
        p = torch.softmax(q[i].double().view(heads, kd) @ seen.T, -1)
        want = p @ seen[:, :rank]
        # weights rounded to 8 bits before their product, the result once more
        assert (out[i].double().view(heads, rank) - want).abs().max() <= 2.0 ** -7 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("tokens", [1, 16, 17, 40, 128, 129])
@pytest.mark.parametrize("heads,n,kk", [(3, 64, 128), (16, 40, 512), (2, 512, 32), (5, 8, 96), (4, 100, 64)])
@pytest.mark.parametrize("gated", [False, True])
def test_products_of_few_rows_per_head(tokens, heads, n, kk, gated):
    from gemmars_b200 import kernels as k
    torch.manual_seed(tokens + n)
    x = torch.randn(tokens, heads, kk + 16, device=DEV).bfloat16()[:, :, 8:8 + kk]
    w = (torch.randn(heads, n, kk, device=DEV) * kk ** -0.5).bfloat16()
    y = torch.zeros(tokens, heads, n + 24, device=DEV, dtype=torch.bfloat16)
    scale = torch.rand(tokens, heads, device=DEV)
    gate = torch.randn(tokens, heads * n + 4, device=DEV)[:, 4:] if gated else None
    k.heads_gemm(x, w, y[:, :, :n], heads, scale=scale, gate=gate)
    want = torch.einsum("thk,hnk->thn", x.double(), w.double()) * scale.double()[..., None]
    if gated:
        want = want * torch.sigmoid(gate.double()).view(tokens, heads, n)
    assert (y[:, :, :n].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 1e-5
    assert not y[:, :, n:].any()
