"""Latent attention over a prompt's own tokens on the tcgen05 kernel: prompts of unequal lengths (sequences that start at no
multiple of eight tokens, tiles and pages that end anywhere), with and without a window, with a gate per head, one per
number and none, against plain sums in 64 bits and against the same layer over the latent rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-6


def _plain(w, h, lens, nh, dim, rot, vd, rank, window, gate):
    out = []
    for x in torch.split(h.double(), lens):
        t = x.shape[0]
        f = (1e4 ** (-torch.arange(0, rot, 2, dtype=torch.float64) / rot)).float().to(DEV)
        a = (torch.arange(t, device=DEV).float()[:, None] * f).double()

        def turn(v):
            c, s = (u.view((t,) + (1,) * (v.dim() - 2) + (-1,)) for u in (torch.cos(a), torch.sin(a)))
            p, q = v[..., 0::2], v[..., 1::2]
            return torch.stack([p * c - q * s, q * c + p * s], -1).flatten(-2)

        m = {k: v.double() for k, v in w.items()}
        q = (x @ m["q"].T).view(t, nh, dim + rot)
        kv = x @ m["dkv"].T
        lat = kv[:, :rank] / torch.sqrt(kv[:, :rank].square().mean(-1, keepdim=True) + EPS) * m["dkv_norm"]
        kr, q = turn(kv[:, rank:]), torch.cat([q[..., :dim], turn(q[..., dim:])], -1) * (dim + rot) ** -0.5
        i = torch.arange(t, device=DEV)
        hide = (i[None] > i[:, None]) | ((i[None] <= i[:, None] - window) if window else torch.zeros(t, t, dtype=torch.bool, device=DEV))
        o = []
        for n in range(nh):
            k = torch.cat([lat @ m["uk"][n * dim:(n + 1) * dim].T, kr], 1)
            p = torch.softmax((q[:, n] @ k.T).masked_fill(hide, -torch.inf), -1)
            o.append(p @ (lat @ m["uv"][n * vd:(n + 1) * vd].T))
        o = torch.stack(o, 1)
        if gate == "channel":
            o = o * torch.sigmoid(x @ m["g"].T).view(t, nh, vd)
        elif gate:
            o = o * torch.sigmoid(x @ m["g"].T)[..., None]
        out.append(o.reshape(t, -1) @ m["o"].T)
    return torch.cat(out)


@pytest.mark.parametrize("lens", [[300], [257, 1, 130, 66], [5, 400, 64], [1030]])
@pytest.mark.parametrize("nh,dim,rot,vd,rank,window,gate", [(3, 128, 64, 128, 512, None, True), (4, 64, 32, 64, 256, 100, "channel"),
                                                            (2, 64, 64, 48, 256, None, False), (2, 128, 8, 16, 256, 70, True)])
def test_prompts_over_expanded_heads(lens, nh, dim, rot, vd, rank, window, gate, monkeypatch):
    from gemmars_b200 import kernels
    assert kernels.latent_prefill_tc_usable(torch.bfloat16, rank, dim, rot, vd)
    _compare(lens, nh, dim, rot, vd, rank, window, gate, monkeypatch)


@pytest.mark.parametrize("nh,dim,rot,vd,rank,window,gate", [(2, 192, 64, 128, 512, None, True), (3, 192, 64, 128, 256, 90, "channel")])
def test_prompts_over_expanded_heads_that_the_tcgen05_kernel_does_not_take(nh, dim, rot, vd, rank, window, gate, monkeypatch):
    """Heads of 192 + 64: rows [v | k_nope | k_rot] on mma.sync."""
    from gemmars_b200 import kernels
    assert not kernels.latent_prefill_tc_usable(torch.bfloat16, rank, dim, rot, vd)
    _compare([257, 1, 130, 66], nh, dim, rot, vd, rank, window, gate, monkeypatch)


def _compare(lens, nh, dim, rot, vd, rank, window, gate, monkeypatch):
    from gemmars_b200 import kernels
    from gemmars_b200.cache.pool import SequenceCache
    from gemmars_b200.parts.base import StepContext, build_part
    from gemmars_b200.parts.plan import PartSpec
    torch.manual_seed(nh + dim + sum(lens))
    hid, t, n = 256, sum(lens), len(lens)
    mat = lambda r, c: (torch.randn(r, c, device=DEV) * c ** -0.5).bfloat16()      # noqa: E731
    w = {"q": mat(nh * (dim + rot), hid) * 2, "dkv": mat(rank + rot, hid), "dkv_norm": torch.randn(rank, device=DEV) * 0.1 + 1,
         "uk": mat(nh * dim, rank), "uv": mat(nh * vd, rank), "o": mat(hid, nh * vd)}
    if gate:
        w["g"] = mat(nh * vd if gate == "channel" else nh, hid)
    part = build_part("mixer", PartSpec("latent_attention", {
        "hidden_size": hid, "num_heads": nh, "dim": dim, "rot_dim": rot, "vdim": vd, "rank": rank, "scale": (dim + rot) ** -0.5,
        "norm_eps": EPS, "gate": gate, "window": window,
        "position": PartSpec("rotary", {"head_dim": rot, "rotary_dim": rot, "theta": 1e4, "layout": "interleaved"})}), "bfloat16")
    part.load(w)
    h = torch.randn(t, hid, device=DEV).bfloat16()
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731

    def run():
        cache = SequenceCache([(0, part.cache_needs())], t + 64 * n, n, 0, max(lens), torch.bfloat16, DEV)
        slots = [cache.open() for _ in lens]
        for s, m in zip(slots, lens):
            cache.extend(s, m)
        cache.sync()
        ctx = StepContext(
            compute="bfloat16", act_dtype=torch.bfloat16, device=torch.device(DEV), n_tokens=t, n_seqs=n,
            tok_pos=ints([j for m in lens for j in range(m)]), tok_seq=ints([i for i, m in enumerate(lens) for _ in range(m)]),
            seq_slot=ints(slots), seq_start=ints([0] * n), seq_len=ints(lens), cu_seqlens=ints([sum(lens[:i]) for i in range(n + 1)]),
            is_decode=False, max_new=max(lens), max_total=max(lens), cache=cache, page_size=64,
            host={"seq_slot": slots, "seq_start": [0] * n, "seq_len": lens})
        rows = torch.zeros(t, hid, device=DEV)
        part.forward(ctx, h, rows, cache.views(0), True)
        kernels.check_status()
        return rows, cache.views(0)[0][1]

    (got, cached), want = run(), _plain(w, h, lens, nh, dim, rot, vd, rank, window, gate)
    # stored activations (queries, keys, values, weights of the softmax, the result) are rounded to 8 bits each
    assert (got.double() - want).norm() <= 8e-3 * want.norm()
    assert (got.double() - want).abs().max() <= 0.06 * want.abs().max()
    monkeypatch.setattr(kernels, "LATENT_EXPAND_MIN_TOKENS", 1 << 30)
    over_rows, cached2 = run()
    assert torch.equal(cached, cached2)                    # the cache is the same whichever way the step takes
    assert (got - over_rows).norm() <= 1.2e-2 * want.norm()
