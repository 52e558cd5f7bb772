"""The row kernels around the recurrences in their prompt forms (several channels a thread, sums on the tensor cores) against
plain sums in 64 bits, at sizes on both sides of what each form takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _packed(lens, slots):
    cu = torch.tensor([0] + lens, device=DEV).cumsum(0).int()
    seq = torch.tensor([i for i, n in enumerate(lens) for _ in range(n)], dtype=torch.int32, device=DEV)
    return cu, seq, torch.tensor(slots, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("lens", [[600], [1, 2, 513, 3, 16, 1], [40, 2, 1]])
@pytest.mark.parametrize("channels", [64, 516, 67, 5124])
@pytest.mark.parametrize("taps,bias,act", [(2, True, True), (3, False, False), (4, True, True), (5, False, True)])
def test_short_filter_of_prompts(lens, channels, taps, bias, act):
    from gemmars_b200 import kernels as k
    torch.manual_seed(channels + taps)
    t, slots = sum(lens), list(range(len(lens)))[::-1]
    cu, seq, slot = _packed(lens, slots)
    wide = torch.randn(t, channels + 8, device=DEV)
    u = wide[:, 4:4 + channels]
    w, b = torch.randn(channels, taps, device=DEV), torch.randn(channels, device=DEV) if bias else None
    state = torch.randn(len(lens) + 1, taps - 1, channels, device=DEV)
    want, kept, at = [], state.double().clone(), 0
    for i, n in enumerate(lens):
        x = torch.cat([state[slots[i]].double(), u[at:at + n].double()])
        y = sum(x[j:j + n] * w[:, j].double() for j in range(taps)) + (b.double() if bias else 0.0)
        want.append(y * torch.sigmoid(y) if act else y)
        kept[slots[i]] = x[x.shape[0] - (taps - 1):]
        at += n
    out = torch.empty(t, channels, device=DEV)
    k.short_filter(u, w, b, state, cu, seq, slot, out, act=act)
    want = torch.cat(want)
    assert (out.double() - want).abs().max() <= 1e-6 * max(1.0, want.abs().max().item()) * taps
    assert torch.equal(state.double(), kept)


@pytest.mark.parametrize("rows,n,group,wn", [(1, 256, 64, 64), (3, 1088, 64, 1088), (7, 2176, 128, 128), (130, 640, 128, 640), (2, 96, 32, 96),
                                              (5, 768, 256, 256), (3, 1536, 512, 1536), (3, 3072, 1024, 3072), (2, 1280, 256, 1280)])
@pytest.mark.parametrize("first,act", [(True, "silu"), (False, "sigmoid")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_gated_norm_of_whole_groups(rows, n, group, wn, first, act, dtype):
    from gemmars_b200 import kernels as k
    torch.manual_seed(n)
    y, gate, w = torch.randn(rows, n, device=DEV) * 3, torch.randn(rows, n + 8, device=DEV), torch.randn(wn, device=DEV)
    for shift in (0, 3):          # rows of the gate at 16-byte boundaries, and not
        g = gate[:, shift:shift + n]
        out = torch.empty(rows, n, device=DEV, dtype=dtype)
        k.gated_group_norm(y, g, w, out, group, 1e-5, first, 0.7, gate_act=act)
        gd = g.double()
        gd = gd * torch.sigmoid(gd) if act == "silu" else torch.sigmoid(gd)
        x = (y.double() * gd if first else y.double()).view(rows, -1, group)
        x = (x / torch.sqrt(x.square().mean(-1, keepdim=True) + 1e-5)).view(rows, n) * w.double().repeat(n // wn)
        want = x * (1.0 if first else gd) * 0.7
        tol = 2e-6 if dtype == torch.float32 else 2.0 ** -8
        assert ((out.double() - want).abs() <= tol * want.abs() + 1e-6).all()


@pytest.mark.parametrize("lens", [[64], [1, 70, 2, 9, 1], [3, 2], [1, 1], [900, 1, 400, 2, 5]])
@pytest.mark.parametrize("channels", [64, 1032, 1100])
def test_mixes_of_prompts(lens, channels):
    from gemmars_b200 import kernels as k
    torch.manual_seed(channels)
    t, slots = sum(lens), list(range(len(lens)))[::-1]
    cu, seq, slot = _packed(lens, slots)
    x, mu = torch.randn(t, channels, device=DEV).bfloat16(), torch.rand(5, channels, device=DEV)
    state = torch.randn(len(lens) + 1, channels, device=DEV)
    before = torch.cat([torch.cat([state[slots[i]][None], x[int(cu[i]):int(cu[i + 1]) - 1].float()]) for i in range(len(lens))])
    want = torch.stack([x.float() + (before - x.float()) * mu[s] for s in range(5)])
    kept = state.clone()
    for i in range(len(lens)):
        kept[slots[i]] = x[int(cu[i + 1]) - 1].float()
    out = k.shift_mix(x, mu, state, cu, seq, slot)
    assert (out.float() - want).abs().max() <= 2.0 ** -8 * want.abs().max()
    assert torch.equal(state, kept)


@pytest.mark.parametrize("rows,channels,rank", [(128, 64, 64), (201, 130, 10), (129, 67, 66), (300, 192, 130), (127, 64, 64), (140, 64, 33)])
@pytest.mark.parametrize("mode", ["tanh_expexp", "rate", "sigmoid_root", "plain"])
def test_low_rank_maps_of_prompts(rows, channels, rank, mode):
    from gemmars_b200 import kernels as k
    torch.manual_seed(rows + rank)
    z = torch.randn(rows, rank + 3, device=DEV)[:, 1:1 + rank]
    w, base = (torch.randn(channels, rank, device=DEV) * rank ** -0.5).bfloat16(), torch.randn(channels, device=DEV)
    zd = z.double()
    a = (torch.tanh(zd) if mode == "tanh_expexp" else zd) @ w.double().T + base.double()
    if mode == "tanh_expexp":
        out, want = k.lowrank_decay(z.contiguous(), w, base), torch.exp(-torch.exp(a))
    elif mode == "rate":
        rate = torch.randn(channels, device=DEV) * 0.5
        out = k.lowrank_map(z, w, base, "rate", rate=rate, rate_group=1)
        want = torch.exp(-torch.exp(rate.double()) * torch.nn.functional.softplus(a))
    elif mode == "sigmoid_root":
        out, want = k.lowrank_map(z, w, base, "sigmoid_root", tau=4.0), torch.sigmoid(a) ** 0.25
    else:
        out, want = k.lowrank_map(z, w, base, "plain"), a
    # a sum of `rank` products rounded to 24 bits each, through functions of slope at most 1 (2.3 for the rates drawn)
    assert (out.double() - want).abs().max() <= 4e-6


@pytest.mark.parametrize("rows,channels,rank", [(2048, 2048, 64), (2011, 2050, 40), (1999, 2003, 33), (1700, 2200, 200)])
@pytest.mark.parametrize("mode", ["tanh_expexp", "rate", "sigmoid_root", "plain"])
def test_low_rank_maps_of_long_prompts_give_the_bits_of_few_tokens(rows, channels, rank, mode):
    """Many tokens by many channels run in tiles, a few tokens by rows: the same sums, infinities included."""
    from gemmars_b200 import kernels as k
    torch.manual_seed(rows + rank)
    z = torch.randn(rows, rank + 3, device=DEV)[:, 1:1 + rank]
    z[rows // 3, 5], z[rows // 2, 7] = float("inf"), float("-inf")
    w, base = (torch.randn(channels, rank, device=DEV) * rank ** -0.5).bfloat16(), torch.randn(channels, device=DEV)
    more = {"rate": torch.randn(channels, device=DEV) * 0.5} if mode == "rate" else {}
    out = k.lowrank_map(z, w, base, mode, tau=4.0, **more)
    for at in (0, rows // 3 - 1, rows // 2 - 2, rows - 3):
        assert torch.equal(k.lowrank_map(z[at:at + 3], w, base, mode, tau=4.0, **more).nan_to_num(7.0), out[at:at + 3].nan_to_num(7.0))
    keep = torch.ones(rows, dtype=torch.bool, device=DEV)
    keep[rows // 3] = keep[rows // 2] = False
    a = (torch.tanh(z.double()) if mode == "tanh_expexp" else z.double()) @ w.double().T + base.double()
    want = {"tanh_expexp": lambda: torch.exp(-torch.exp(a)), "sigmoid_root": lambda: torch.sigmoid(a) ** 0.25, "plain": lambda: a,
            "rate": lambda: torch.exp(-torch.exp(more["rate"].double()) * torch.nn.functional.softplus(a))}[mode]()
    # a sum of `rank` products rounded to 24 bits each, through functions of slope at most 1 (2.3 for the rates drawn)
    assert (out.double() - want)[keep].abs().max() <= 6e-6
