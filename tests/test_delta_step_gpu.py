"""A gated delta layer's single tokens in one kernel: the bits of the filter, the recurrence and the norm one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,groups,dim,vdim,taps", [(4, 2, 128, 128, 4), (8, 2, 64, 64, 2), (3, 3, 128, 64, 8), (2, 1, 36, 128, 3),
                                                        (4, 1, 20, 64, 4), (2, 2, 100, 128, 5)])
@pytest.mark.parametrize("seqs", [1, 5])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_the_bits_of_the_kernels_one_by_one(heads, groups, dim, vdim, taps, seqs, dtype):
    from gemmars_b200 import kernels as k
    assert k.delta_step_usable(seqs, seqs, heads, groups, dim, vdim, taps)
    g = torch.Generator(device="cuda").manual_seed(heads * dim + seqs)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")       # noqa: E731
    qk, hv = groups * dim, heads * vdim
    c, width = 2 * qk + hv, 2 * qk + 2 * hv + 2 * heads
    wide, filt = r(seqs, width + 8 - width % 4), r(c, taps)      # rows at 16-byte boundaries: the norm's wide form
    a_log, dt_bias, norm = r(heads).abs().log(), r(heads), r(vdim)
    slots = torch.tensor([(3 * i + 1) % 7 for i in range(seqs)], dtype=torch.int32, device="cuda")
    states = [(r(8, taps - 1, c), r(8, heads, k.recurrent_state_floats(dim, vdim)))]
    states.append(tuple(s.clone() for s in states[0]))
    cu = torch.arange(seqs + 1, dtype=torch.int32, device="cuda")
    seq = torch.arange(seqs, dtype=torch.int32, device="cuda")
    outs = [torch.empty(seqs, hv, device="cuda", dtype=dtype) for _ in range(2)]
    for step in range(3):                # on what the step before has left
        proj = (wide.roll(step, 0) * (1 + 0.1 * step))[:, :width]
        fs, st = states[0]
        f, y = torch.empty(seqs, c, device="cuda"), torch.empty(seqs, hv, device="cuda")
        k.short_filter(proj[:, :c], filt, None, fs, cu, seq, slots, f, act=True)
        k.delta_rule(f[:, :qk], f[:, qk:2 * qk], f[:, 2 * qk:], proj[:, c + hv:c + hv + heads], proj[:, c + hv + heads:], a_log, dt_bias, st,
                     cu, slots, y, heads, groups, dim, vdim, dim ** -0.5)
        k.gated_group_norm(y, proj[:, c:c + hv], norm, outs[0], vdim, 1e-6, False, 0.7)
        k.delta_step(proj, filt, states[1][0], a_log, dt_bias, states[1][1], slots, norm, outs[1], heads, groups, dim, vdim, dim ** -0.5,
                     1e-6, 0.7)
        assert torch.equal(outs[0], outs[1])
        assert torch.equal(states[0][0], states[1][0])
        # the decay's zero rows beyond the head's dims stay what they were times the decay in both
        assert torch.equal(states[0][1], states[1][1])


def test_what_is_refused_runs_as_before():
    from gemmars_b200 import kernels as k
    assert not k.delta_step_usable(5, 4, 4, 2, 128, 128, 4)          # a prompt among them
    assert not k.delta_step_usable(4, 4, 4, 1, 128, 128, 4)          # sixteen blocks a q/k head
    assert not k.delta_step_usable(4, 4, 4, 2, 256, 128, 4)
    assert not k.delta_step_usable(4, 4, 4, 2, 128, 96, 4)
    assert not k.delta_step_usable(4, 4, 4, 2, 128, 128, 1)


def _layer(heads, groups, dim, vdim, hidden=64, conv=4):
    from gemmars_b200.csrc import build
    from gemmars_b200.parts.base import build_part
    from gemmars_b200.parts.plan import PartSpec
    part = build_part("mixer", PartSpec("gated_delta", {"hidden_size": hidden, "heads": heads, "kv_heads": groups, "dim": dim, "vdim": vdim,
                                                        "conv": conv, "norm_eps": 1e-6}), "float32")
    build.ensure(part.kernel_units())
    g = torch.Generator(device="cuda").manual_seed(heads * dim)
    part.load({n: torch.randn(w.shape, generator=g, device="cuda") * (w.shape[-1] ** -0.5 if len(w.shape) == 2 else 0.5)
               for n, w in part.wants().items()})
    return part


@pytest.mark.parametrize("heads,groups,dim,vdim", [(3, 3, 128, 64), (1, 1, 33, 64), (5, 5, 64, 128), (4, 2, 128, 128)])
def test_a_token_alone_has_the_bits_of_the_same_token_among_many(heads, groups, dim, vdim):
    """Rows of a layer's own width, which are at 16-byte boundaries or not: one sequence may take the one kernel, many do not."""
    from gemmars_b200.cache.pool import SequenceCache
    from gemmars_b200.parts.base import StepContext
    part = _layer(heads, groups, dim, vdim)
    many = 150
    g = torch.Generator(device="cuda").manual_seed(7)
    h = torch.randn(many, 64, generator=g, device="cuda")
    past = [torch.randn(s.shape, generator=g, device="cuda") for s in part.cache_needs()]
    ints = lambda v: torch.tensor(list(v), dtype=torch.int32, device="cuda")       # noqa: E731
    rows, states = [], []
    for n in (1, many):
        cache = SequenceCache([(0, part.cache_needs())], 64 * many, n, 0, 64, torch.float32, torch.device("cuda"))
        for _ in range(n):
            cache.extend(cache.open(), 1)
        cache.sync()
        caches = cache.views(0)
        for c, p in zip(caches, past):
            c[:n] = p
        ctx = StepContext(compute="float32", act_dtype=torch.float32, device=torch.device("cuda"), n_tokens=n, n_seqs=n, tok_pos=ints([0] * n),
                          tok_seq=ints(range(n)), seq_slot=ints(range(n)), seq_start=ints([0] * n), seq_len=ints([1] * n),
                          cu_seqlens=ints(range(n + 1)), is_decode=True, max_new=1, max_total=1, cache=cache, page_size=64, host=None)
        out = torch.zeros(n, 64, device="cuda")
        part.forward(ctx, h[:n], out, caches)
        rows.append(out[0])
        states.append([c[0].clone() for c in caches])
    assert torch.equal(*rows)
    assert all(torch.equal(a, b) for a, b in zip(*states))


def test_rows_that_the_norm_sums_in_another_order_are_refused():
    from gemmars_b200 import kernels as k
    assert k.delta_step_usable(1, 1, 4, 2, 128, 128, 4, 2 * 256 + 2 * 512 + 8)
    assert not k.delta_step_usable(1, 1, 3, 3, 128, 64, 4, 2 * 384 + 2 * 192 + 6)        # rows
    assert not k.delta_step_usable(1, 1, 1, 1, 33, 64, 4, 2 * 33 + 2 * 64 + 2)           # the gate's place in them


def _both(seqs, slots, heads, groups, dim, vdim, taps=4):
    """Outputs and states of the three kernels and of the one, from the same past."""
    from gemmars_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(seqs)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")       # noqa: E731
    qk, hv, n_slots = groups * dim, heads * vdim, max(slots) + 1
    c, width = 2 * qk + hv, 2 * qk + 2 * hv + 2 * heads
    proj, filt = r(seqs, width + -width % 4)[:, :width], r(c, taps)
    a_log, dt_bias, norm = r(heads).abs().log(), r(heads), r(vdim)
    fs, st = r(n_slots, taps - 1, c), r(n_slots, heads, k.recurrent_state_floats(dim, vdim))
    slots = torch.tensor(slots, dtype=torch.int32, device="cuda")
    cu = torch.arange(seqs + 1, dtype=torch.int32, device="cuda")
    made = []
    for one in (False, True):
        f1, s1, out = fs.clone(), st.clone(), torch.empty(seqs, hv, device="cuda")
        if one:
            k.delta_step(proj, filt, f1, a_log, dt_bias, s1, slots, norm, out, heads, groups, dim, vdim, dim ** -0.5, 1e-6, 1.0)
        else:
            f, y = torch.empty(seqs, c, device="cuda"), torch.empty(seqs, hv, device="cuda")
            k.short_filter(proj[:, :c], filt, None, f1, cu, cu[:-1], slots, f, act=True)
            k.delta_rule(f[:, :qk], f[:, qk:2 * qk], f[:, 2 * qk:], proj[:, c + hv:c + hv + heads], proj[:, c + hv + heads:], a_log, dt_bias, s1,
                         cu, slots, y, heads, groups, dim, vdim, dim ** -0.5)
            k.gated_group_norm(y, proj[:, c:c + hv], norm, out, vdim, 1e-6, False)
        made.append((out, f1, s1))
    return made


@pytest.mark.parametrize("heads,groups,dim,vdim,per_sm", [(8, 4, 128, 128, 3), (4, 4, 64, 64, 6), (16, 8, 32, 64, 6)])
def test_as_many_blocks_as_there_is_room_for(heads, groups, dim, vdim, per_sm):
    from gemmars_b200 import kernels as k
    most = per_sm * k.sm_count() // (heads * vdim // 32)
    assert k.delta_step_usable(most, most, heads, groups, dim, vdim, 4) and not k.delta_step_usable(most + 1, most + 1, heads, groups, dim, vdim, 4)
    apart, one = _both(most, list(range(most)), heads, groups, dim, vdim)
    assert all(torch.equal(a, b) for a, b in zip(apart, one))


def test_rows_that_pad_a_captured_step_share_a_slot():
    """Three rows on the spare slot: the others' outputs and states are what they are without them."""
    apart, one = _both(7, [2, 0, 5, 1, 6, 6, 6], 4, 2, 128, 128)
    for a, b in zip(apart, one):
        rows = [0, 1, 2, 3] if a.shape[0] == 7 and a.dim() == 2 else [0, 1, 2, 5]
        assert torch.equal(a[rows], b[rows])
