"""The rows that a prompt expands per head: every sequence from a multiple of 8 on, the same numbers as the copy token by
token, zeros where no token lies, whatever was there."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [(1,), (7, 8, 9), (16, 1, 23, 64), (15, 15)])
@pytest.mark.parametrize("heads,dim,rd,rank,half", [(9, 64, 32, 256, False), (16, 128, 64, 512, False), (3, 64, 16, 1040, True), (8, 64, 0, 32, False)])
def test_rows_to_expand(lens, heads, dim, rd, rank, half):
    from gemmars_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(sum(lens) + rank)
    t, n = sum(lens), len(lens)
    q = torch.randn(t, heads * (dim + rd), generator=g, device="cuda")
    kv = torch.randn(t, rank + rd, generator=g, device="cuda")
    gate_in = torch.randn(t, heads, generator=g, device="cuda")
    w = torch.rand(rank, generator=g, device="cuda") + 0.5
    inv = (1.0 / (1e4 ** (torch.arange(rd // 2, dtype=torch.float64) / max(1, rd // 2)))).float().cuda() if rd else None
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")       # noqa: E731
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    pos, seq, slots = ints([i for m in lens for i in range(m)]), ints([b for b, m in enumerate(lens) for _ in range(m)]), ints(list(range(n)))
    table = ints([list(range(b * 2 + 1, b * 2 + 3)) for b in range(n)])
    cache = [torch.zeros(2 * n + 1, 64, rank + rd, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    qn, qr = (torch.empty(t, heads * d, device="cuda", dtype=torch.bfloat16) for d in (dim, rank + rd))
    dense = torch.empty(t, rank + rd, device="cuda", dtype=torch.bfloat16)
    gates = [torch.empty(t, heads, device="cuda") for _ in range(2)]
    k.latent_prepare(q, kv, gate_in, w, 1e-6, inv, rd, 0.3, qn, qr, gates[0], cache[0], table, 64, pos, seq, slots, heads, dim, rd, rank,
                     dense=dense, half_layout=half)
    rows = k.latent_expand_rows(t, n)
    lat, keys = (torch.full((rows, d), float("nan"), device="cuda", dtype=torch.bfloat16) for d in (rank, rd))
    both = torch.empty(t, heads * (dim + rd), device="cuda", dtype=torch.bfloat16)
    k.latent_prepare(q, kv, gate_in, w, 1e-6, inv, rd, 0.3, both, both, gates[1], cache[1], table, 64, pos, seq, slots, heads, dim, rd, rank,
                     half_layout=half, expand=(lat, keys, ints(cu)))
    at = torch.tensor([(cu[b] // 8 + b) * 8 + i for b, m in enumerate(lens) for i in range(m)], device="cuda")
    want = torch.zeros(rows, rank + rd, device="cuda", dtype=torch.bfloat16)
    want[at] = dense
    assert torch.equal(lat, want[:, :rank]) and torch.equal(keys, want[:, rank:])
    assert torch.equal(cache[0], cache[1]) and torch.equal(gates[0], gates[1])
    both = both.view(t, heads, dim + rd)
    assert torch.equal(both[:, :, :dim], qn.view(t, heads, dim)) and torch.equal(both[:, :, dim:], qr.view(t, heads, rank + rd)[:, :, rank:])
    x = kv[:, :rank].double()
    ref = x / (x.square().mean(1, keepdim=True) + 1e-6).sqrt() * w.double()
    assert ((dense[:, :rank].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-6).all()
