"""Routed experts against plain sums in 64 bits where the two bfloat16 paths change their ways: a few tokens by expert (one
pass of 8 or 16 entries and several, runs of rows and pieces of the inner dimension that end inside a block, sizes that go
token by token instead), and prompts in padded tiles of 128 and 256 rows whose counts end anywhere (also experts that nobody
or everybody chose)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(t, e, top, width, ff, ffs, skew, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)     # noqa: E731
    z = rand(t, e)
    z[:, :top] += skew
    idx = z.topk(top, dim=1).indices.int().contiguous()
    wts = torch.softmax(rand(t, top), 1).contiguous()
    m = {"h": rand(t, width).bfloat16(), "gu": (rand(e, 2 * ff, width) * width ** -0.5).bfloat16(), "d": (rand(e, width, ff) * ff ** -0.5).bfloat16()}
    if ffs:
        m.update(sgu=(rand(2 * ffs, width) * width ** -0.5).bfloat16(), sd=(rand(width, ffs) * ffs ** -0.5).bfloat16(), sg=torch.rand(t, generator=g, device=DEV))
    return idx, wts, m, rand(t, width)


def _gated(x, w, lim, wt=1.0):
    a, b = (x @ w.double().T * wt).chunk(2, -1)
    a, b = a.clamp(max=lim), b.clamp(-lim, lim)
    return a * torch.sigmoid(1.7 * a) * (b + 0.5)


def _add(out, room, y, d, scale):
    out += y @ d.double().T * scale
    room += y.abs() @ d.double().abs().T * scale


def _want(idx, wts, m, lim, weigh_input, plain=None):
    """The sums, and what rounding the middle to 8 bits can move them by."""
    x = m["h"].double()
    out, room = torch.zeros_like(x), torch.zeros_like(x)
    for e in range(m["d"].shape[0]):
        t, s = (idx == e).nonzero(as_tuple=True)
        wt = wts[t, s].double()[:, None]
        w = m["gu"][e]
        if plain:
            y = x[t] @ w.double().T
            y = torch.relu(y) ** 2 if plain == "relu2" else torch.nn.functional.gelu(y)
        else:
            y = _gated(x[t], w, lim, wt if weigh_input else 1.0)
        o, r = torch.zeros_like(x[t]), torch.zeros_like(x[t])
        _add(o, r, y, m["d"][e], 1.0 if weigh_input and not plain else wt)
        out.index_add_(0, t, o)
        room.index_add_(0, t, r)
    if "sg" in m:
        _add(out, room, _gated(x, m["sgu"], 2.0), m["sd"], m["sg"].double()[:, None])
    return out, 2.0 ** -8 * room + 1e-4 * room.max()


def _run(kernels, idx, wts, m, base, lim, weigh_input, run, rows=slice(None)):
    res = base[rows].clone()
    run(m["h"][rows], idx[rows].contiguous(), wts[rows].contiguous(), m["sg"][rows].contiguous() if "sg" in m else None, m["gu"], m["d"], m.get("sgu"),
        m.get("sd"), res, lim, 2.0, 1.7, 0.5, weigh_input=weigh_input)
    kernels.check_status()
    return res


@pytest.mark.parametrize("tokens", [1, 2, 8, 9, 15, 40])
@pytest.mark.parametrize("e,top,width,ff,ffs,skew", [(8, 2, 64, 32, 0, 0.), (5, 5, 96, 160, 96, 0.), (64, 6, 256, 96, 64, 8.), (9, 1, 544, 40, 24, 0.),
                                                     (3, 2, 72, 64, 0, 4.)])
def test_few_tokens(tokens, e, top, width, ff, ffs, skew):
    from gemmars_b200 import kernels
    idx, wts, m, base = _case(tokens, e, top, width, ff, ffs, skew, tokens + e)
    for weigh in (False, True):
        got = _run(kernels, idx, wts, m, base, 1.5, weigh, kernels.moe_experts)
        want, room = _want(idx, wts, m, 1.5, weigh)
        assert ((got.double() - base.double() - want).abs() <= room).all()
        for t in (0, tokens - 1):          # alone as in the batch
            assert torch.equal(_run(kernels, idx, wts, m, base, 1.5, weigh, kernels.moe_experts, slice(t, t + 1))[0], got[t])


@pytest.mark.parametrize("tokens", [1, 7, 12])
@pytest.mark.parametrize("act", ["gelu", "relu2"])
@pytest.mark.parametrize("width,ff", [(96, 64), (64, 72), (256, 200)])
def test_few_tokens_without_a_gate(tokens, act, width, ff):
    from gemmars_b200 import kernels
    idx, wts, m, base = _case(tokens, 6, 3, width, ff, 0, 1.0, tokens + ff)
    m["gu"] = m["gu"][:, :ff].contiguous()
    got = base.clone()
    kernels.moe_experts_plain(m["h"], idx, wts, m["gu"], m["d"], got, act=act)
    want, room = _want(idx, wts, m, 1.0, False, act)
    assert ((got.double() - base.double() - want).abs() <= room).all()


@pytest.mark.parametrize("tokens", [16, 33, 100, 256, 331, 1030])
@pytest.mark.parametrize("e,top,width,ff,ffs,skew", [(2, 2, 128, 64, 64, 0.), (64, 6, 256, 128, 0, 0.), (40, 2, 136, 64, 0, 9.), (7, 3, 128, 192, 128, 3.)])
@pytest.mark.parametrize("weigh", [False, True])
def test_prompts_in_padded_tiles(tokens, e, top, width, ff, ffs, skew, weigh):
    from gemmars_b200 import kernels
    idx, wts, m, base = _case(tokens, e, top, width, ff, ffs, skew, tokens + e)
    assert kernels.moe_tc_usable(m["h"], m["gu"], m["d"])
    got = _run(kernels, idx, wts, m, base, 1.5, weigh, kernels.moe_experts_tc)
    want, room = _want(idx, wts, m, 1.5, weigh)
    assert ((got.double() - base.double() - want).abs() <= room).all()


@pytest.mark.parametrize("rows", [65, 100, 300, 2048])
@pytest.mark.parametrize("n", [1, 65, 130, 576, 1000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_products_of_few_features_in_narrow_tiles(rows, n, dtype):
    """The tile's width changes nothing: the same bits as in tiles of 256 rows."""
    from gemmars_b200 import kernels
    torch.manual_seed(rows + n)
    x, w = torch.randn(rows, 328, device=DEV).bfloat16(), torch.randn(n, 328, device=DEV).bfloat16()
    got, wide = torch.full((rows, n), 7.0, device=DEV, dtype=dtype), torch.full((rows, n), 7.0, device=DEV, dtype=dtype)
    kernels.gemm_tc_persistent(x, w, got)
    kernels.gemm_tc_persistent(x, w, wide, bn=256)
    kernels.check_status()
    assert torch.equal(got, wide)
    want = x.double() @ w.double().T       # float32 sums of 328 products, then the result's own rounding
    assert (got.double() - want).abs().max() <= (2.0 ** -8 if dtype is torch.bfloat16 else 1e-5) * want.abs().max()


@pytest.mark.parametrize("features", [8, 24, 100, 2056])
def test_the_shared_experts_activation(features):
    from gemmars_b200 import kernels
    torch.manual_seed(features)
    gu, scale = torch.randn(33, 2 * features, device=DEV).bfloat16() * 3, torch.rand(33, device=DEV)
    y = torch.empty(33, features, device=DEV, dtype=torch.bfloat16)
    f = kernels._fn("grouped_gemm", "gb_gated_act", [kernels.c_void_p] * 3 + [kernels.c_int] * 2 + [kernels.c_float] * 3 + [kernels.c_void_p])
    assert f(gu.data_ptr(), y.data_ptr(), scale.data_ptr(), 33, features, 2.0, 1.7, 0.5, kernels._stream()) == 0
    g, u = gu.double().chunk(2, 1)
    g, u = g.clamp(max=2.0), u.clamp(-2.0, 2.0)
    want = g * torch.sigmoid(1.7 * g) * (u + 0.5) * scale.double()[:, None]
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all()
