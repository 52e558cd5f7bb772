"""The recurrences of a prompt taken in chunks of 16 tokens against plain sums in 64 bits, token by token, and against the
kernels that walk token by token: borders of chunks, sequences shorter than one, sizes that fill no tile, decays of zero,
states carried in and out, and heads taken in turns."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LENS = [100, 1, 16, 33, 15, 64, 17]
SLOTS = [3, 1, 6, 0, 7, 2, 5]


def _plain(q, k, v, g, new, bonus, S):
    """(outputs, state) of one head: q, k, g [n, dim], v [n, vdim]; ``new`` [n] the delta rule's beta, or None."""
    out = []
    for t in range(q.shape[0]):
        if bonus is not None:
            out.append(q[t] @ S + (q[t] * bonus * k[t]).sum() * v[t])
            S = g[t][:, None] * S + torch.outer(k[t], v[t])
            continue
        S = g[t][:, None] * S
        S = S + torch.outer(k[t], v[t] if new is None else new[t] * (v[t] - k[t] @ S))
        out.append(q[t] @ S)
    return torch.stack(out), S


@pytest.mark.parametrize("turns", [False, True])
@pytest.mark.parametrize("heads,groups,dim,vdim", [(4, 2, 128, 128), (2, 1, 64, 64), (3, 3, 12, 33), (6, 2, 100, 20), (40, 20, 128, 40),
                                                    (24, 12, 128, 128), (48, 24, 100, 72)])      # the last two: over 1,184 groups of 16 columns
@pytest.mark.parametrize("form", ["delta", "channel_delta", "ssd", "before", "after"])
def test_chunks_of_a_prompt(form, heads, groups, dim, vdim, turns, monkeypatch):
    from gemmars_b200 import kernels as k
    if turns and heads > 8:
        pytest.skip("the small sizes show it")
    if turns:
        monkeypatch.setattr(k, "CHUNK_SCAN_SCRATCH", 1)         # one head at a time
    gen = torch.Generator().manual_seed(heads * 1000 + dim + vdim)
    ntok, gh = sum(LENS), groups if form in ("delta", "channel_delta", "ssd") else heads
    rand = lambda *s: torch.randn(s, generator=gen)      # noqa: E731
    x = rand(ntok, 2 * gh * dim + heads * vdim + 4)
    gates = rand(ntok, 2 * heads + 1) * 2
    a_log, dt_bias, skip, bonus = rand(heads) * 0.5, rand(heads) * 0.5, rand(heads), rand(heads, dim)
    decay = torch.exp(-torch.exp(rand(ntok, heads * dim) * 2 - 2))
    decay[5, :] = 0.0
    decay[40, ::2] = 0.0
    start = rand(len(LENS), heads, dim, vdim)
    lanes = 1 if dim <= 32 else 2 if dim <= 64 else 4
    full = torch.zeros(len(LENS), heads, 32 * lanes, vdim)
    full[:, :, :dim] = start
    stored = full.view(-1, heads, lanes, 8, 4, vdim).permute(0, 1, 3, 5, 2, 4).reshape(len(LENS), heads, -1)
    state = torch.zeros(9, heads, k.recurrent_state_floats(dim, vdim))
    for i, s in enumerate(SLOTS):
        state[s] = stored[i]
    q, kk, v = (t.double() for t in (x[:, :gh * dim], x[:, gh * dim:2 * gh * dim], x[:, 2 * gh * dim:2 * gh * dim + heads * vdim]))
    q, kk, v = q.view(ntok, gh, dim), kk.view(ntok, gh, dim), v.view(ntok, heads, vdim)
    z, rate, new = gates.double(), torch.exp(a_log.double()), None
    soft = torch.nn.functional.softplus
    if form in ("delta", "channel_delta"):
        q, kk = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, kk))
        q, new = q * dim ** -0.5, torch.sigmoid(z[:, :heads])
    g = decay.double().view(ntok, heads, dim)
    if form == "delta":
        g = torch.exp(-rate * soft(z[:, heads:2 * heads] + dt_bias.double()))[..., None].expand(ntok, heads, dim)
    if form == "ssd":
        dt = soft(z[:, :heads] + dt_bias.double())
        g, new = torch.exp(-rate * dt)[..., None].expand(ntok, heads, dim), None
    rep = heads // gh
    want, final, at = torch.zeros(ntok, heads, vdim, dtype=torch.float64), torch.zeros(len(LENS), heads, dim, vdim, dtype=torch.float64), 0
    for i, n in enumerate(LENS):
        for h in range(heads):
            r = slice(at, at + n)
            kh = kk[r, h // rep] * (dt[r, h, None] if form == "ssd" else 1.0)
            o, final[i, h] = _plain(q[r, h // rep], kh, v[r, h], g[r, h], None if new is None else new[r, h],
                                    bonus[h].double() if form == "before" else None, start[i, h].double())
            want[r, h] = o + (skip[h].double() * v[r, h] if form == "ssd" else 0.0)
        at += n
    dev = lambda t: t.to(DEV)      # noqa: E731
    xd, gd, cu = dev(x), dev(gates), dev(torch.tensor([0] + LENS).cumsum(0).int())
    slots, dd = dev(torch.tensor(SLOTS, dtype=torch.int32)), dev(decay)
    a, b, c = xd[:, :gh * dim], xd[:, gh * dim:2 * gh * dim], xd[:, 2 * gh * dim:2 * gh * dim + heads * vdim]

    def run(chunked):
        st, y = dev(state).clone(), torch.empty(ntok, heads * vdim, device=DEV)
        if form == "delta":
            k.delta_rule(a, b, c, gd[:, :heads], gd[:, heads:2 * heads], dev(a_log), dev(dt_bias), st, cu, slots, y, heads, groups, dim,
                         vdim, dim ** -0.5, chunked=chunked)
        elif form == "channel_delta":
            k.channel_delta_rule(a, b, c, gd[:, :heads], dd, st, cu, slots, y, heads, groups, dim, vdim, dim ** -0.5, chunked=chunked)
        elif form == "ssd":
            k.ssd_scan(c, b, a, gd[:, :heads], dev(a_log), dev(dt_bias), dev(skip), st, cu, slots, y, heads, groups, dim, vdim,
                       chunked=chunked)
        else:
            k.wkv_scan(a, b, dd, c, dev(bonus) if form == "before" else None, st, cu, slots, y, heads, dim, vdim, 0.5, chunked=chunked)
        held = st[slots.long()].cpu().view(len(LENS), heads, 8, vdim, lanes, 4).permute(0, 1, 4, 2, 5, 3).reshape(len(LENS), heads, -1, vdim)
        assert not st[4].any() and not st[8].any()          # slots of no sequence of the step
        assert not held[:, :, dim:].any()
        scale = 0.5 if form in ("before", "after") else 1.0
        off = lambda u, w: ((u.double() - w).norm() / w.norm()).item()      # noqa: E731
        return off(y.cpu().view(ntok, heads, vdim), want * scale), off(held[:, :, :dim], final)

    (y_err, s_err), (y_walk, s_walk) = run(True), run(False)
    # a few roundings of 2^-24 an element, and what the split products leave out (2^-21 of a product at most, of either sign)
    assert y_err < 1.5e-6 and s_err < 1.5e-6, (y_err, s_err, y_walk, s_walk)


@pytest.mark.parametrize("heads,groups,dim,vdim", [(4, 2, 128, 128), (2, 1, 64, 64), (3, 3, 12, 33), (40, 20, 128, 40), (24, 12, 128, 128)])
@pytest.mark.parametrize("form", ["delta", "channel_delta", "ssd", "before", "after"])
@pytest.mark.parametrize("what", ["q", "k", "v", "gate"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_number_that_is_not_finite_reaches_what_it_reaches_token_by_token(form, heads, groups, dim, vdim, what, value):
    """Tokens before it keep their bits, and what is not finite afterwards is what is not finite token by token."""
    from gemmars_b200 import kernels as k
    torch.manual_seed(heads + dim)
    lens, bad = [100, 40, 3, 1, 17, 20, 33, 16], (37, 104, 175)       # inside a chunk, near a sequence's start, near the end of one
    ntok, gh = sum(lens), groups if form in ("delta", "channel_delta", "ssd") else heads
    x = torch.randn(ntok, 2 * gh * dim + heads * vdim + 4, device=DEV)
    gates, decay = torch.randn(ntok, 2 * heads, device=DEV), torch.exp(-torch.exp(torch.randn(ntok, heads * dim, device=DEV) - 1))
    a_log, dt_bias, skip, bonus = (torch.randn(s, device=DEV) * 0.5 for s in ((heads,), (heads,), (heads,), (heads, dim)))
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    slots = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    start = torch.zeros(len(lens), heads, k.recurrent_state_floats(dim, vdim), device=DEV)

    def run(x, gates, decay, chunked):
        a, b, c = x[:, :gh * dim], x[:, gh * dim:2 * gh * dim], x[:, 2 * gh * dim:2 * gh * dim + heads * vdim]
        st, y = start.clone(), torch.empty(ntok, heads * vdim, device=DEV)
        if form == "delta":
            k.delta_rule(a, b, c, gates[:, :heads], gates[:, heads:], a_log, dt_bias, st, cu, slots, y, heads, groups, dim, vdim,
                         dim ** -0.5, chunked=chunked)
        elif form == "channel_delta":
            k.channel_delta_rule(a, b, c, gates[:, :heads], decay, st, cu, slots, y, heads, groups, dim, vdim, dim ** -0.5, chunked=chunked)
        elif form == "ssd":
            k.ssd_scan(c, b, a, gates[:, :heads], a_log, dt_bias, skip, st, cu, slots, y, heads, groups, dim, vdim, chunked=chunked)
        else:
            k.wkv_scan(a, b, decay, c, bonus if form == "before" else None, st, cu, slots, y, heads, dim, vdim, 1.0, chunked=chunked)
        return y, st

    clean, _ = run(x, gates, decay, True)
    assert clean.isfinite().all()
    x, gates, decay = x.clone(), gates.clone(), decay.clone()
    for t in bad:
        if what == "gate":
            gates[t, 0] = gates[t, heads] = float("nan")
            decay[t, 1] = float("nan")
        else:
            x[t, {"q": 0, "k": gh * dim, "v": 2 * gh * dim}[what] + 2] = value
    (y, st), (y_walk, st_walk) = run(x, gates, decay, True), run(x, gates, decay, False)
    for i, at in enumerate(cu[:-1].tolist()):
        first = min([t for t in bad if at <= t < at + lens[i]], default=at + lens[i])
        assert torch.equal(y[at:first], clean[at:first]), i
    assert torch.equal(y.isfinite(), y_walk.isfinite()) and torch.equal(st.isfinite(), st_walk.isfinite())
    assert not y.isfinite().all()


@pytest.mark.parametrize("ntok,nseq,dims", [(1, 1, 1), (16, 1, 64), (17, 3, 65), (2048, 1, 128), (1000, 40, 100)])
@pytest.mark.parametrize("delta", [False, True])
def test_scratch_of_a_step(ntok, nseq, dims, delta):
    """The size that the step works out is the library's."""
    import ctypes
    from gemmars_b200 import kernels as k
    from gemmars_b200.csrc import build
    f = build.load("recurrent_chunk").gb_chunk_floats
    f.restype = ctypes.c_longlong
    assert f(ntok, nseq, dims, int(delta)) == k.chunk_floats(ntok, nseq, dims, delta)


@pytest.mark.parametrize("heads,dim,vdim", [(4, 128, 128), (3, 64, 64), (2, 100, 40)])
@pytest.mark.parametrize("form", ["ssd", "before", "after"])
def test_sums_of_one_sign_are_not_cut(form, heads, dim, vdim):
    """A state that 1,000 tokens only add to: its numbers are off by roundings of either sign.  The tensor core's cut of every sum
    would make them 0.72 x 2^-24 (4.3e-8) and more too small on the mean, a cut operand 2^-24; token by token the mean is below 1e-8."""
    from gemmars_b200 import kernels as k
    torch.manual_seed(dim)
    ntok, lanes = 1000, 2 if dim <= 64 else 4
    x = torch.rand(ntok, heads * (2 * dim + vdim), device=DEV) + 0.5
    a, b, c = x[:, :heads * dim], x[:, heads * dim:2 * heads * dim], x[:, 2 * heads * dim:]
    cu, slots = torch.tensor([0, ntok], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    one = torch.ones(ntok, heads * dim, device=DEV)
    steps, a_log = torch.rand(ntok, heads, device=DEV), torch.full((heads,), -60.0, device=DEV)      # exp(-e^-60 dt) is 1
    for chunked in (True, False):
        st, y = torch.zeros(1, heads, k.recurrent_state_floats(dim, vdim), device=DEV), torch.empty(ntok, heads * vdim, device=DEV)
        scale = 1.0
        if form == "ssd":
            zero = torch.zeros(heads, device=DEV)
            k.ssd_scan(c, b, a, steps, a_log, zero, zero, st, cu, slots, y, heads, heads, dim, vdim, chunked=chunked)
            scale = torch.nn.functional.softplus(steps).double()[:, :, None]       # as the kernel has them, in float32
        else:
            k.wkv_scan(a, b, one, c, torch.ones(heads, dim, device=DEV) if form == "before" else None, st, cu, slots, y, heads, dim, vdim,
                       1.0, chunked=chunked)
        held = st[0].view(heads, 8, vdim, lanes, 4).permute(0, 3, 1, 4, 2).reshape(heads, -1, vdim)[:, :dim]
        want = torch.einsum("thd,thv->hdv", b.double().reshape(ntok, heads, dim) * scale, c.double().reshape(ntok, heads, vdim))
        off = (held.double() / want - 1.0).mean().item()
        assert abs(off) < 2e-8, (chunked, off)
