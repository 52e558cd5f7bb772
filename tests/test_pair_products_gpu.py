"""Prompt products worked by pairs of CTAs, at the edges of their tiles: half a pair beyond the result, tokens and inner
elements that end within a tile, narrower tiles, parts of the inner dimension, groups narrower than a tile."""
from ctypes import c_int

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def k():
    from gemmars_b200 import kernels
    return kernels


def pairs(k, m, n, kk, bn, ctas, gated=False):
    return k._fn("gemm_tc", "gb_gemm_tc_pairs", [c_int] * 6)(m, n, kk, bn, ctas, int(gated))


def operands(m, n, kk, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(m, kk, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, kk, generator=g, device="cuda") * kk ** -0.5).bfloat16()
    return x, w


def exact_and_bound(x, w):
    """The product in 64 bits and a bound on what float32 sums may be off: an ulp of the largest partial sum per addition."""
    xd, wd = x.double(), w.double()
    return xd @ wd.T, x.shape[1] * 2.0 ** -23 * (xd.abs() @ wd.abs().T)


@pytest.mark.parametrize("m,n,kk,bn", [(1000, 1664, 200, None), (500, 128, 4104, None), (2048, 1196, 64, None), (700, 392, 1032, 160),
                                       (257, 1280, 520, 256), (600, 768, 136, 144)])
def test_plain_and_adding_products(k, m, n, kk, bn):
    assert pairs(k, m, n, kk, bn or 256, 4) == 1
    x, w = operands(m, n, kk, m + n)
    bias = torch.randn(n, device="cuda")
    want, bound = exact_and_bound(x, w)
    y = torch.full((m, n), 7.0, device="cuda")
    k.gemm_tc_persistent(x, w, y, bias, bn=bn, ctas=4)
    assert ((y.double() - want - bias.double()).abs() <= bound + 2.0 ** -22 * (want.abs() + 4)).all()
    start = torch.randn(m, n, device="cuda")
    for split in (False, True):
        y = start.clone()
        k.gemm_tc_persistent(x, w, y, accumulate=True, bn=bn, ctas=4, split_last=split)
        assert ((y.double() - want - start.double()).abs() <= bound + 2.0 ** -21 * (want.abs() + 8)).all()
    y16 = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    k.gemm_tc_persistent(x, w, y16, bn=bn, ctas=4)
    assert ((y16.double() - want).abs() <= bound + 2.0 ** -8 * (want.abs() + bound)).all()
    assert k.gemm_tc_status() == 0


@pytest.mark.parametrize("m,n,kk", [(520, 192, 200), (1000, 72, 4104), (300, 960, 64), (520, 188, 200), (1000, 1672, 72)])
def test_gated_product(k, m, n, kk):
    """Also results whose features are no multiple of 8 (a box of W's rows at a time) or end within a warp's 16."""
    assert pairs(k, m, n, kk, 256, 4, True) == 1
    x, w = operands(m, 2 * n, kk, m + n)
    y = torch.empty(m, n, device="cuda", dtype=torch.bfloat16)
    k.gemm_tc_persistent(x, w, y, swiglu=True, ctas=4)
    one = torch.empty_like(y)
    k.gemm_tc_persistent(x, w, one, swiglu=True, ctas=1)          # one CTA walks all tiles: never a pair
    narrow = torch.empty_like(y)
    k.gemm_tc_persistent(x, w, narrow, swiglu=True, bn=112, ctas=4)   # tiles that end after half of a round's tokens
    g, u = (x.double() @ w[:n].double().T), (x.double() @ w[n:].double().T)
    want = g * torch.sigmoid(g) * u
    # bfloat16's half step, and the two sums' float32 errors through a slope of at most 1.1 |u| and 1.1 |g|
    _, bound = exact_and_bound(x, w)
    tol = 2.0 ** -8 * want.abs() + 1.2 * (u.abs() * bound[:, :n] + (g.abs() + 1) * bound[:, n:]) + 2.0 ** -20 * (g.abs() + 1) * (u.abs() + 1)
    assert ((y.double() - want).abs() <= tol).all() and ((one.double() - want).abs() <= tol).all() and ((narrow.double() - want).abs() <= tol).all()
    assert k.gemm_tc_status() == 0


@pytest.mark.parametrize("nh,nkv,lengths", [(3, 1, (300, 77)), (4, 1, (513,)), (2, 0, (1000,))])
def test_qkv_product_is_the_single_ctas(k, nh, nkv, lengths):
    """An odd number of heads leaves half of the last pair beyond the result."""
    m, kk, n = sum(lengths), 264, (nh + 2 * nkv) * 128
    assert pairs(k, m, n, kk, 256, 4) == 1
    x, w = operands(m, n, kk, m)
    tok_pos = torch.tensor([i for l in lengths for i in range(l)], dtype=torch.int32, device="cuda")
    tok_seq = torch.tensor([q for q, l in enumerate(lengths) for _ in range(l)], dtype=torch.int32, device="cuda")
    slots = torch.arange(len(lengths), dtype=torch.int32, device="cuda")
    width = max(-(-l // 64) for l in lengths)
    table = (torch.arange(len(lengths) * width, dtype=torch.int32, device="cuda") + 1).view(len(lengths), width)
    inv = (1.0 / (1e4 ** (torch.arange(64, dtype=torch.float64) / 64.0))).float().cuda()
    qw = torch.rand(128, device="cuda") + 0.5
    got = []
    for ctas in (1, 4):
        kc = torch.zeros((len(lengths) * width + 1, max(nkv, 1), 64, 128), device="cuda", dtype=torch.bfloat16)
        vc = torch.zeros((len(lengths) * width + 1, max(nkv, 1), 128, 64), device="cuda", dtype=torch.bfloat16)
        q = torch.full((m, nh * 128), 9.0, device="cuda", dtype=torch.bfloat16)
        k.gemm_qkv_prompt(x, w, None, q, nh, nkv, 128, qw, qw, 1e-6, k.rope_table(tok_pos, inv), 0.1,
                          k.token_place(tok_pos, tok_seq, slots, table, 64) if nkv else None, 64, kc if nkv else None,
                          vc if nkv else None, ctas=ctas)
        got.append((q, kc, vc))
    for a, b in zip(*got):       # the same products up to float32 sums: a bfloat16 step where those straddle a rounding
        assert ((a.float() - b.float()).abs() <= 2.0 ** -7 * a.float().abs() + 1e-5).all()
    assert k.gemm_tc_status() == 0


@pytest.mark.parametrize("counts", [(1, 0, 33, 255, 256, 300), (16, 17, 0, 0, 511, 64)])
def test_groups_narrower_than_a_tile(k, monkeypatch, counts):
    n, kk, bn, e = 480, 200, 256, len(counts)
    monkeypatch.setattr(k, "sm_count", lambda device=None: 4)
    tile_expert, tile_rows = [], []
    for g, c in enumerate(counts):
        for first in range(0, c, bn):
            tile_expert.append(g)
            tile_rows.append(min(bn, c - first))
    tile_expert += [-1, -1]
    tile_rows += [0, 0]
    rows = len(tile_expert) * bn
    assert pairs(k, rows, n, kk, bn, 4) == 1 and pairs(k, rows, n, kk, bn, 4, True) == 1
    x, w = operands(rows, e * 2 * n, kk, 5)
    te, tr = (torch.tensor(v, dtype=torch.int32, device="cuda") for v in (tile_expert, tile_rows))
    scale = torch.rand(rows, device="cuda") + 0.5
    y = torch.zeros(rows, n, device="cuda")
    k.gemm_tc_grouped(x, w.view(2 * e * n, kk)[:e * n].contiguous(), y, n, e, te, bn=bn, tile_rows=tr)
    yg = torch.zeros(rows, n, device="cuda", dtype=torch.bfloat16)
    k.gemm_tc_grouped(x, w, yg, n, e, te, scale, gated=True, bn=bn, tile_rows=tr)
    for t, (g, c) in enumerate(zip(tile_expert, tile_rows)):
        if c == 0:
            continue
        xs, at = x[t * bn:t * bn + c], slice(t * bn, t * bn + c)
        want, bound = exact_and_bound(xs, w[g * n:(g + 1) * n])
        assert ((y[at].double() - want).abs() <= bound + 2.0 ** -22 * want.abs()).all()
        wg = w[2 * g * n:2 * (g + 1) * n]
        a, u = xs.double() @ wg[:n].double().T, xs.double() @ wg[n:].double().T
        want = a * torch.sigmoid(a) * u * scale[at, None].double()
        _, bound = exact_and_bound(xs, wg)
        tol = 2.0 ** -8 * want.abs() + 1.8 * (u.abs() * bound[:, :n] + (a.abs() + 1) * bound[:, n:]) + 2.0 ** -19 * (a.abs() + 1) * (u.abs() + 1)
        assert ((yg[at].double() - want).abs() <= tol).all()
    assert k.gemm_tc_status() == 0


@pytest.mark.parametrize("t,width,ffs", [(129, 64, 72), (300, 200, 1024), (2048, 264, 320), (511, 128, 2816)])
def test_shared_expert_with_its_activation_in_the_product(k, t, width, ffs):
    x, w = operands(t, 2 * ffs, width, t)
    down = (torch.randn(width, ffs, device="cuda") * ffs ** -0.5).bfloat16()
    sg, residual = torch.rand(t, device="cuda"), torch.randn(t, width, device="cuda")
    got = residual.clone()
    k._shared_expert(x, sg, w, down, got, 1.5, 1.702, 1.0)
    g, u = (x.double() @ w[:ffs].double().T).clamp(max=1.5), (x.double() @ w[ffs:].double().T).clamp(-1.5, 1.5)
    act = g * torch.sigmoid(1.702 * g) * (u + 1) * sg[:, None].double()
    want = residual.double() + act @ down.double().T
    # an activation is rounded to bfloat16 once; what float32 sums and the clamps' edges add is far below its half step
    tol = (2.0 ** -8 * act.abs() + 1e-4) @ down.double().abs().T + 2.0 ** -21 * (want.abs() + 4)
    assert ((got.double() - want).abs() <= tol).all()
    assert k.gemm_tc_status() == 0


@pytest.mark.parametrize("sms", [4, 3, None])
@pytest.mark.parametrize("groups,t,n,kk", [(4, 65, 200, 136), (3, 300, 384, 72), (2, 513, 128, 264), (4, 256, 1000, 64), (5, 270, 130, 4104)])
def test_a_batch_of_products(k, monkeypatch, sms, groups, t, n, kk):
    """Groups that start at any row: a tile's last piece of tokens ends at its group's last row."""
    if sms:
        monkeypatch.setattr(k, "sm_count", lambda device=None: sms)
    x, w = operands(groups * t, groups * n, kk, t)
    out = torch.full((groups, t, n), 7.0, device="cuda")
    k.gemm_batch(x.view(groups, t, kk), w.view(groups, n, kk), out)
    for g in range(groups):
        want, bound = exact_and_bound(x[g * t:(g + 1) * t], w[g * n:(g + 1) * n])
        assert ((out[g].double() - want).abs() <= bound + 2.0 ** -22 * want.abs()).all()
    assert k.gemm_tc_status() == 0


def test_one_round_of_tiles_takes_pairs_where_they_are_the_faster(k):
    """Both sides measured: up to 4,096 inner elements a single round is the faster with one CTA a tile."""
    for m, n, kk, paired in ((2048, 2048, 4096, 0), (1000, 4096, 4096, 0), (700, 4096, 6144, 1), (2048, 2048, 6144, 1), (2048, 4096, 4096, 1),
                             (2048, 4672, 2048, 0)):
        assert pairs(k, m, n, kk, 256, 148) == paired


def test_a_product_without_groups_refuses_what_belongs_to_groups(k):
    x, w = operands(256, 128, 64, 1)
    y = torch.empty(256, 128, device="cuda")
    tile_rows = torch.full((1,), 256, dtype=torch.int32, device="cuda")
    with pytest.raises(AssertionError):
        k.gemm_tc_grouped(x, w, y, 128, 1, None, tile_rows=tile_rows, bn=256)
    with pytest.raises(AssertionError):
        k.gemm_tc_grouped(x, w, y, 128, 1, None, torch.ones(255, device="cuda"), bn=256)
