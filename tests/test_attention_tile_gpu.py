"""Plain attention of prompts with sixteen queries a block: the bits of one token a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,lens,starts,window", [
    (16, 8, 128, (75, 90, 136), (0, 0, 0), None), (16, 8, 100, (129, 31), (70, 3), None), (32, 8, 64, (95,), (257,), None),
    (24, 8, 32, (150, 1), (0, 300), None), (20, 20, 36, (131,), (5,), None), (16, 8, 128, (300,), (0,), 290)])
def test_the_bits_of_one_token_a_block(dtype, nh, nkv, hd, lens, starts, window):
    from gemmars_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(hd + nh)
    t, n = sum(lens), len(lens)
    width = max(-(-(s + m) // 64) for s, m in zip(starts, lens))
    table = (torch.randperm(n * width, generator=torch.Generator().manual_seed(1)) + 1).to(torch.int32).view(n, width).cuda()
    kc = torch.randn(n * width + 1, nkv, 64, hd, generator=g, device="cuda").to(dtype)
    vc = torch.randn(n * width + 1, nkv, hd, 64, generator=g, device="cuda").to(dtype)
    q = (torch.randn(t, nh * hd, generator=g, device="cuda") * hd ** -0.5).to(dtype)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")       # noqa: E731
    pos, seq = ints([s + i for s, m in zip(starts, lens) for i in range(m)]), ints([b for b, m in enumerate(lens) for _ in range(m)])
    outs = []
    for apart in (True, False):
        outs.append(torch.empty_like(q))
        k.attention_ref(q, outs[-1], nh, kc, vc, table, 64, pos, seq, ints(list(range(n))), window, apart=apart)
    assert torch.equal(*outs) and torch.isfinite(outs[0].float()).all()
    at = t - 1                                   # the last token of the last sequence against 64 bits
    end = starts[-1] + lens[-1]
    pages = table[-1].long()
    keys = kc[pages].permute(0, 2, 1, 3).reshape(-1, nkv, hd)[:end].double()
    values = vc[pages].permute(0, 3, 1, 2).reshape(-1, nkv, hd)[:end].double()
    lo = max(0, end - window) if window else 0
    qd = q[at].view(nkv, nh // nkv, hd).double()
    w = torch.softmax(torch.einsum("ghd,kgd->ghk", qd, keys[lo:]), dim=-1)
    want = torch.einsum("ghk,kgd->ghd", w, values[lo:]).reshape(-1)
    assert (outs[1][at].double() - want).abs().max() <= (1e-5 if dtype == torch.float32 else 2.0 ** -8 * want.abs().max() + 1e-5)


@pytest.mark.parametrize("nh,nkv,hd", [(16, 8, 128), (12, 12, 64), (24, 6, 40)])
@pytest.mark.parametrize("lens,starts,window", [((130, 1, 1, 1, 1, 1, 3, 2), (0, 300, 20, 0, 129, 128, 7, 250), None), ((90, 1, 70, 1), (0, 200, 30, 5), 64)])
def test_forms_and_mixed_steps(nh, nkv, hd, lens, starts, window):
    """One token, four tokens and sixteen queries a block over a step in which neighbours share nothing: the same bits."""
    from gemmars_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(hd)
    t, n = sum(lens), len(lens)
    width = max(-(-(s + m) // 64) for s, m in zip(starts, lens))
    table = (torch.randperm(n * width, generator=torch.Generator().manual_seed(1)) + 1).to(torch.int32).view(n, width).cuda()
    kc, vc = torch.randn(n * width + 1, nkv, 64, hd, generator=g, device="cuda"), torch.randn(n * width + 1, nkv, hd, 64, generator=g, device="cuda")
    q = torch.randn(t, nh * hd, generator=g, device="cuda") * hd ** -0.5
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")       # noqa: E731
    pos, seq = ints([s + i for s, m in zip(starts, lens) for i in range(m)]), ints([b for b, m in enumerate(lens) for _ in range(m)])
    outs = []
    for form in (1, 4, 16, 0):
        outs.append(torch.full_like(q, 9.0))
        k.attention_ref(q, outs[-1], nh, kc, vc, table, 64, pos, seq, ints(list(range(n))), window, apart=False, form=form)
    assert all(torch.equal(outs[0], o) for o in outs[1:]) and torch.isfinite(outs[0]).all()
