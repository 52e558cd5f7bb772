"""The calls this framework is timed on: single layers and short models, through the entry points a program uses.

A layer is a part of the registry (``build_part``) run as the step function runs it: the batch of a step described by a
``StepContext``, keys and states in a ``SequenceCache``, prompt steps launched one after the other, steps of single tokens
replayed from a captured graph.  The two ``qwen`` kinds are whole calls of ``Runner.step`` on models of a few layers.
Sizes are those of the framework's own configurations (``tuning.py``: the Qwen3 shapes and the pairs small, lite, mid).
"""
import math

import torch

from gemmars_b200 import Engine, kernels  # noqa: F401  (the package registers its parts and architectures)
from gemmars_b200.cache.pool import SequenceCache
from gemmars_b200.csrc import build
from gemmars_b200.engine.step import Runner, StepItem
from gemmars_b200.parts.base import StepContext, build_part
from gemmars_b200.parts.plan import PartSpec

DEV = "cuda:0"
EPS = 1e-6

SIZES = {  # layer widths of the framework's pairs, and the Qwen3 shapes of like width
    "small": {"hidden": 1024, "heads": 8, "window": 512, "inter": 3072, "qwen_heads": 16, "latent_heads": 8, "rank": 256,
              "latent_dim": 64, "latent_rot": 32, "latent_vdim": 64, "experts": 16, "top": 2, "ff": 512, "shared": 1024},
    "lite": {"hidden": 2048, "heads": 16, "window": 1024, "inter": 6144, "qwen_heads": 16, "latent_heads": 16, "rank": 512,
             "latent_dim": 128, "latent_rot": 64, "latent_vdim": 128, "experts": 64, "top": 6, "ff": 1408, "shared": 2816},
    "mid": {"hidden": 4096, "heads": 32, "window": 2048, "inter": 12288, "qwen_heads": 32, "latent_heads": 32, "rank": 512,
            "latent_dim": 128, "latent_rot": 64, "latent_vdim": 128, "experts": 32, "top": 4, "ff": 2048, "shared": 4096},
}
VOCAB = 151936


def listed():
    return [
        # one more token for each of eight conversations of 8,192 tokens: the framework's headline decode, four layers of it
        {"name": "qwen_step", "kind": "qwen", "size": "mid", "dtype": "bfloat16", "layers": 4, "seqs": 8, "tokens": 1, "context": 8191},
        # a prompt of 2,048 tokens of the same sizes, two layers, to the next token's logits
        {"name": "qwen_prompt", "kind": "qwen", "size": "mid", "dtype": "bfloat16", "layers": 2, "seqs": 1, "tokens": 2048, "context": 0},
        # the true 32-bit path, which results are checked against: three short prompts of unequal lengths in one step
        {"name": "qwen_prompt_f32", "kind": "qwen", "size": "small", "dtype": "float32", "layers": 2, "seqs": 3, "tokens": 301, "context": 0},
        # delta-rule layer, prompt of 2,048 tokens
        {"name": "delta_prompt", "kind": "delta", "size": "mid", "dtype": "bfloat16", "seqs": 1, "tokens": 2048, "context": 0},
        # the same layer for one more token of one conversation: the smallest call, where latency counts
        {"name": "delta_step", "kind": "delta", "size": "lite", "dtype": "bfloat16", "seqs": 1, "tokens": 1, "context": 700},
        # state-space layer, four prompts of unequal lengths that start together
        {"name": "ssd_prompts", "kind": "ssd", "size": "lite", "dtype": "bfloat16", "seqs": 4, "tokens": 1901, "context": 0},
        # linear attention with a decay per channel, prompt of 2,048 tokens
        {"name": "wkv_prompt", "kind": "wkv", "size": "mid", "dtype": "bfloat16", "seqs": 1, "tokens": 2048, "context": 0},
        # windowed attention with a cap, a filter and a gate: one more token for eight conversations of 4,096 tokens
        {"name": "capped_step", "kind": "capped", "size": "mid", "dtype": "bfloat16", "seqs": 8, "tokens": 1, "context": 4096},
        # latent attention, prompt of 2,048 tokens
        {"name": "latent_prompt", "kind": "latent", "size": "lite", "dtype": "bfloat16", "seqs": 1, "tokens": 2048, "context": 0},
        # latent attention, one more token for sixteen conversations of up to 8,192 tokens
        {"name": "latent_step", "kind": "latent", "size": "lite", "dtype": "bfloat16", "seqs": 16, "tokens": 1, "context": 8000},
        # routed feed-forward beside a shared one, prompt of 2,048 tokens
        {"name": "moe_prompt", "kind": "moe", "size": "lite", "dtype": "bfloat16", "seqs": 1, "tokens": 2048, "context": 0},
        # the same for one more token of eight conversations
        {"name": "moe_step", "kind": "moe", "size": "lite", "dtype": "bfloat16", "seqs": 8, "tokens": 1, "context": 1000},
    ]


def _spread(rng, low, high):
    """A whole number between ``low`` and ``high``, spread evenly over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(("qwen", "delta", "delta", "ssd", "wkv", "capped", "latent", "moe"))
    case = {"kind": kind, "size": rng.choice(("small", "lite", "mid")), "dtype": "bfloat16"}
    if kind == "qwen":
        case["layers"] = rng.randint(1, 2)
        if rng.random() < 0.3:
            case.update(size="small", dtype="float32")
    if kind == "ssd" or kind == "moe" and case["size"] == "mid":
        case["size"] = rng.choice(("small", "lite"))
    if rng.random() < 0.5 and case["dtype"] == "bfloat16":           # single tokens
        seqs = _spread(rng, 1, 32)
        case.update(seqs=seqs, tokens=1, context=_spread(rng, 100, min(8191, 65536 // seqs)))
    else:
        tokens = _spread(rng, 40, 400 if case["dtype"] == "float32" else 2048)
        case.update(seqs=rng.randint(1, 4), tokens=tokens, context=0)
    return case


# ---------------------------------------------------------------- what a case is made of

def _lens(case):
    """Tokens that each sequence brings: one, or unequal shares of the step's tokens."""
    n = case["seqs"]
    if case["tokens"] == 1:
        return [1] * n
    whole = n * (n + 1) // 2
    lens = [max(1, case["tokens"] * (i + 1) // whole) for i in range(n)]
    lens[-1] += case["tokens"] - sum(lens)
    return lens


def _starts(case):
    """Tokens that each sequence has behind it: the context, shorter by up to a third from one sequence to the last
    (equal where the batch is eight, as in the framework's benchmark)."""
    n, c = case["seqs"], case["context"]
    return [c if n == 8 else c - c * i // (3 * n) for i in range(n)]


def _is_step(case):
    return case["tokens"] == 1


class _Rand:
    def __init__(self, seed, case):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 1000003 + 17)
        self.act = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def n(self, *shape, std=1.0, mean=0.0):
        return torch.randn(shape, generator=self.g, device=DEV) * std + mean

    def u(self, low, high, *shape):
        return torch.rand(shape, generator=self.g, device=DEV) * (high - low) + low

    def w(self, rows, cols):
        """A matrix in the compute type: rows of unit-variance results for inputs of unit variance."""
        return self.n(rows, cols, std=cols ** -0.5).to(self.act)


def _dims(case):
    z = SIZES[case["size"]]
    return {"hidden": z["hidden"], "nh": z["heads"], "nkv": z["heads"] // 2, "ssd_heads": 2 * z["heads"],
            "groups": max(1, z["heads"] // 4), "wkv_heads": z["hidden"] // 64}


def _part(case):
    """(category, kind, parameters) of the layer's part."""
    z, d, h = SIZES[case["size"]], _dims(case), SIZES[case["size"]]["hidden"]
    kind = case["kind"]
    if kind == "delta":
        return "mixer", "gated_delta", {"hidden_size": h, "heads": d["nh"], "kv_heads": d["nkv"], "dim": 128, "vdim": 128,
                                        "conv": 4, "norm_eps": EPS}
    if kind == "ssd":
        return "mixer", "ssd", {"hidden_size": h, "heads": d["ssd_heads"], "vdim": 64, "state": 128, "groups": d["groups"],
                                "norm_groups": d["groups"], "conv": 4, "norm_eps": EPS}
    if kind == "wkv":
        return "mixer", "wkv", {"hidden_size": h, "heads": d["wkv_heads"], "dim": 64, "rank": 64, "norm_eps": EPS}
    if kind == "capped":
        return "mixer", "capped_attention", {
            "hidden_size": h, "heads": z["heads"], "kv_heads": z["heads"] // 4, "dim": 128, "vdim": 128, "bias": True, "conv": 3,
            "window": z["window"], "scale": 128 ** -0.5, "softcap": 30.0, "gate": True,
            "position": PartSpec("rotary", {"head_dim": 128, "rotary_dim": 128, "theta": 1e6, "layout": "half"})}
    if kind == "latent":
        return "mixer", "latent_attention", {
            "hidden_size": h, "num_heads": z["latent_heads"], "dim": z["latent_dim"], "rot_dim": z["latent_rot"],
            "vdim": z["latent_vdim"], "rank": z["rank"], "scale": (z["latent_dim"] + z["latent_rot"]) ** -0.5, "norm_eps": EPS,
            "gate": True, "window": None,
            "position": PartSpec("rotary", {"head_dim": z["latent_rot"], "rotary_dim": z["latent_rot"], "theta": 1e4,
                                            "layout": "interleaved"})}
    assert kind == "moe"
    return "ffn", "moe", {"hidden_size": h, "experts": z["experts"], "top": z["top"], "ff": z["ff"], "limit": 7.0, "alpha": 1.702,
                          "shift": 1.0, "router_bias": True, "shared": {"ff": z["shared"], "limit": 7.0, "gate": True}}


def _tensors(case, r):
    """The part's tensors by its short names."""
    z, d, h = SIZES[case["size"]], _dims(case), SIZES[case["size"]]["hidden"]
    kind = case["kind"]

    def rates(n):       # decay rates of 1 to 16 and step sizes of 0.001 to 0.1
        dt = torch.exp(r.u(math.log(1e-3), math.log(1e-1), n))
        return {"A_log": torch.log(r.u(1.0, 16.0, n)), "dt_bias": dt + torch.log(-torch.expm1(-dt))}

    if kind == "delta":
        qk, hv = d["nkv"] * 128, d["nh"] * 128
        return {"q": r.w(qk, h), "k": r.w(qk, h), "v": r.w(hv, h), "g": r.w(hv, h), "b": r.w(d["nh"], h), "a": r.w(d["nh"], h),
                "o": r.w(h, hv), "q_conv": r.n(qk, 4, std=0.4), "k_conv": r.n(qk, 4, std=0.4), "v_conv": r.n(hv, 4, std=0.4),
                "norm": r.n(128, std=0.1, mean=1.0), **rates(d["nh"])}
    if kind == "ssd":
        inner, gn = d["ssd_heads"] * 64, d["groups"] * 128
        return {"in": r.w(2 * inner + 2 * gn + d["ssd_heads"], h), "o": r.w(h, inner), "conv": r.n(inner + 2 * gn, 4, std=0.4),
                "conv_bias": r.n(inner + 2 * gn, std=0.02), "D": r.n(d["ssd_heads"], std=0.1, mean=1.0),
                "norm": r.n(inner, std=0.1, mean=1.0), **rates(d["ssd_heads"])}
    if kind == "wkv":
        w = {"mu_" + s: r.u(0.0, 1.0, h) for s in "rkvgw"}
        w.update({s: r.w(h, h) for s in "rkvgo"})
        w.update({"w1": r.w(64, h), "w2": r.n(h, 64, std=0.05).to(r.act), "w0": r.u(-6.0, -0.5, h),
                  "u": r.n(d["wkv_heads"], 64, std=0.3, mean=0.3), "norm": r.n(h, std=0.1, mean=1.0)})
        return w
    if kind == "capped":
        nq, nk = z["heads"] * 128, z["heads"] // 4 * 128
        w = {"q": r.w(nq, h), "k": r.w(nk, h), "v": r.w(nk, h), "g": r.w(nq, h), "o": r.w(h, nq)}
        for s, n in (("q", nq), ("k", nk), ("v", nk)):
            w[s + "_bias"], w[s + "_conv"] = r.n(n, std=0.02), r.n(n, 3, std=0.4)
        return w
    if kind == "latent":
        nh, dim, rot, vd, rank = z["latent_heads"], z["latent_dim"], z["latent_rot"], z["latent_vdim"], z["rank"]
        return {"q": r.w(nh * (dim + rot), h), "dkv": r.w(rank + rot, h), "dkv_norm": r.n(rank, std=0.1, mean=1.0),
                "uk": r.w(nh * dim, rank), "uv": r.w(nh * vd, rank), "o": r.w(h, nh * vd), "g": r.w(nh, h)}
    ff, sf = z["ff"], z["shared"]
    w = {"router": r.w(z["experts"], h), "router_bias": r.n(z["experts"], std=0.1)}
    for e in range(z["experts"]):
        w.update({f"e{e}.gate": r.w(ff, h), f"e{e}.up": r.w(ff, h), f"e{e}.down": r.w(h, ff)})
    w.update({"shared.gate": r.w(sf, h), "shared.up": r.w(sf, h), "shared.down": r.w(h, sf), "shared.sg": r.w(1, h)})
    return w


def _made(case, seed):
    """What a layer's call has: its tensors, the normed activations, the residual stream, and what the sequences left."""
    r, z, d, h = _Rand(seed, case), SIZES[case["size"]], _dims(case), SIZES[case["size"]]["hidden"]
    t = sum(_lens(case))
    # a stream no larger than what the layer adds to it, so that the outputs show the layer
    m = {"w": _tensors(case, r), "h": r.n(t, h).to(r.act), "x": r.n(t, h, std=0.05), "past": {}}
    if not any(_starts(case)):
        return m
    n, kind = case["seqs"], case["kind"]
    if kind == "delta":
        m["past"] = {"filter": r.n(n, 3, (2 * d["nkv"] + d["nh"]) * 128), "S": r.n(n, d["nh"], 128, 128, std=0.3)}
    elif kind == "ssd":
        m["past"] = {"filter": r.n(n, 3, d["ssd_heads"] * 64 + 2 * d["groups"] * 128), "S": r.n(n, d["ssd_heads"], 128, 64, std=0.3)}
    elif kind == "wkv":
        m["past"] = {"filter": r.n(n, h).to(r.act).float(), "S": r.n(n, d["wkv_heads"], 64, 64, std=0.3)}
    elif kind == "capped":
        nk, seen = z["heads"] // 4, [min(s, z["window"]) for s in _starts(case)]     # older keys are out of every window
        m["past"] = {"filter": r.n(n, 2, (z["heads"] + 2 * nk) * 128), "k": [r.n(s, nk, 128).to(r.act) for s in seen],
                     "v": [r.n(s, nk, 128).to(r.act) for s in seen]}
    elif kind == "latent":
        m["past"] = {"rows": [r.n(s, z["rank"] + z["latent_rot"]).to(r.act) for s in _starts(case)]}
    return m


def _state_order(S):
    """[n, heads, dims, cols] in the order a state lies in memory: 32 dims to a lane, four of them side by side."""
    n, nh, dims, cols = S.shape
    lanes = 1 if dims <= 32 else 2 if dims <= 64 else 4 if dims <= 128 else 8
    return S.reshape(n, nh, lanes, 8, 4, cols).permute(0, 1, 3, 5, 2, 4).reshape(n, nh, -1)


def _into_pages(group, layer, slot, first, k, v):
    """Writes a sequence's keys (and values) of positions ``first`` .. into the pages the cache gave it."""
    pos = torch.arange(first, first + k.shape[0], device=DEV)
    page = group.page_table[slot][(pos // group.page_size) % group.table_width].long()
    kc, vc = group.layer(layer)
    kc[page, :, pos % group.page_size] = k
    if v is not None:
        vc[page, :, :, pos % group.page_size] = v


# ---------------------------------------------------------------- one layer

class _Layer:
    """A part with its cache and the batch of one step, as the step function sets them up."""

    def __init__(self, case, made):
        category, kind, params = _part(case)
        self.case, self.ffn = case, category == "ffn"
        self.part = build_part(category, PartSpec(kind, params), case["dtype"])
        build.ensure(self.part.kernel_units())
        self.part.load(made["w"])
        self.h, self.x, self.rows = made["h"], made["x"], torch.empty_like(made["x"])
        lens, starts = _lens(case), _starts(case)
        n, t = len(lens), sum(lens)
        self.cache = SequenceCache([(0, self.part.cache_needs())] if self.part.cache_needs() else [],
                                   sum(s + m + 64 for s, m in zip(starts, lens)), n, 0, max(64, max(lens)), self.h.dtype, DEV)
        slots = [self.cache.open() for _ in range(n)]
        for slot, s, m in zip(slots, starts, lens):
            if s:
                self.cache.extend(slot, s)
            self.cache.extend(slot, m)
        self.cache.sync()
        self.caches = self.cache.views(0)
        past = made["past"]
        for i, slot in enumerate(slots):
            if "filter" in past:
                self.caches[1 if case["kind"] == "capped" else 0][slot] = past["filter"][i]
            if "S" in past:
                self.caches[1][slot] = _state_order(past["S"][i:i + 1])[0]
            if "k" in past:
                k = past["k"][i]
                _into_pages(self.caches[0][0], 0, slot, starts[i] - k.shape[0], k, past["v"][i])
            if "rows" in past:
                _into_pages(self.caches[0][0], 0, slot, 0, past["rows"][i][:, None], None)
        self.states = [c[:n] for c in self.caches if torch.is_tensor(c)]
        seq = [i for i, m in enumerate(lens) for _ in range(m)]
        pos = [s + j for s, m in zip(starts, lens) for j in range(m)]
        cu = [0]
        for m in lens:
            cu.append(cu[-1] + m)

        def ints(v):
            return torch.tensor(v, dtype=torch.int32, device=DEV)

        self.ctx = StepContext(
            compute=case["dtype"], act_dtype=self.h.dtype, device=torch.device(DEV), n_tokens=t, n_seqs=n, tok_pos=ints(pos),
            tok_seq=ints(seq), seq_slot=ints(slots), seq_start=ints(starts), seq_len=ints(lens), cu_seqlens=ints(cu),
            is_decode=_is_step(case), max_new=max(lens), max_total=max(s + m for s, m in zip(starts, lens)), cache=self.cache,
            page_size=self.cache.page_size,
            host=None if _is_step(case) else {"seq_slot": slots, "seq_start": starts, "seq_len": lens})
        self.graph = None

    def once(self):
        self.ctx.extras.clear()
        self.rows.copy_(self.x)
        build.set_pdl(True)
        try:
            if self.ffn:
                self.part.forward(self.ctx, self.h, self.rows)
            else:
                self.part.forward(self.ctx, self.h, self.rows, self.caches, True)
        finally:
            build.set_pdl(False)

    def capture(self):
        kept = [s.clone() for s in self.states]
        self.once()
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.once()
        for s, k in zip(self.states, kept):
            s.copy_(k)


# ---------------------------------------------------------------- whole models

def _qwen_config(case):
    z = SIZES[case["size"]]
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": case["layers"],
            "hidden_size": z["hidden"], "num_attention_heads": z["qwen_heads"], "num_key_value_heads": 8, "head_dim": 128,
            "intermediate_size": z["inter"], "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": EPS,
            "attention_bias": False, "tie_word_embeddings": case["size"] == "small", "max_position_embeddings": 40960}


def _qwen_made(case, seed):
    r, z = _Rand(seed, case), SIZES[case["size"]]
    h, inter, nq, nk = z["hidden"], z["inter"], z["qwen_heads"] * 128, 8 * 128

    def norm(n):
        return r.n(n, std=0.1, mean=1.0)

    def table():
        t = torch.empty((VOCAB, h), dtype=r.act, device=DEV)
        for a in range(0, VOCAB, 16384):
            t[a:a + 16384] = r.n(min(16384, VOCAB - a), h, std=0.02)
        return t

    w = {"model.embed_tokens.weight": table(), "model.norm.weight": norm(h)}
    if case["size"] != "small":
        w["lm_head.weight"] = table()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w.update({p + "input_layernorm.weight": norm(h), p + "post_attention_layernorm.weight": norm(h),
                  p + "self_attn.q_proj.weight": r.w(nq, h), p + "self_attn.k_proj.weight": r.w(nk, h),
                  p + "self_attn.v_proj.weight": r.w(nk, h), p + "self_attn.o_proj.weight": r.w(h, nq),
                  p + "self_attn.q_norm.weight": norm(128), p + "self_attn.k_norm.weight": norm(128),
                  p + "mlp.gate_proj.weight": r.w(inter, h), p + "mlp.up_proj.weight": r.w(inter, h),
                  p + "mlp.down_proj.weight": r.w(h, inter)})
    t = sum(_lens(case))
    ids = torch.randint(0, VOCAB, (t,), generator=r.g, device=DEV)
    past = [[(r.n(s, 8, 128).to(r.act), r.n(s, 8, 128).to(r.act)) for s in _starts(case) if s] for _ in range(case["layers"])]
    return w, ids, past


class _Qwen:
    """A model in an engine's runner, its sequences open, and the tokens of the step."""

    def __init__(self, case, seed):
        w, ids, past = _qwen_made(case, seed)
        lens, starts = _lens(case), _starts(case)
        self.case = case
        self.engine = Engine.from_config(_qwen_config(case), w, {
            "dtype": case["dtype"], "max_batch": case["seqs"], "max_tokens": sum(s + m + 128 for s, m in zip(starts, lens))})
        self.runner = self.engine.runner
        ids, at, self.tokens = ids.tolist(), 0, []
        for m in lens:
            self.tokens.append(ids[at:at + m])
            at += m
        self.slots, self.starts = [], starts
        if _is_step(case):
            cache = self.runner.cache
            self.slots = [self.runner.open() for _ in starts]
            for slot, s in zip(self.slots, starts):
                cache.extend(slot, s)
            cache.sync()
            for layer in range(case["layers"]):
                for i, slot in enumerate(self.slots):
                    _into_pages(cache.kv_groups[0], layer, slot, 0, *past[layer][i])

    def step(self):
        r = self.runner
        if _is_step(self.case):         # a token is run, and taken back afterwards as after a draft that is refused
            out = r.step([StepItem(s, t, [0]) for s, t in zip(self.slots, self.tokens)])
            for s, n in zip(self.slots, self.starts):
                r.cache.truncate(s, n)
            return out
        slots = [r.open() for _ in self.tokens]
        out = r.step([StepItem(s, t, [len(t) - 1]) for s, t in zip(slots, self.tokens)])
        for s in reversed(slots):
            r.close(s)
        return out


# ---------------------------------------------------------------- the interface

def prepare(case, seed):
    if case["kind"] == "qwen":
        return _Qwen(case, seed)
    layer = _Layer(case, _made(case, seed))
    if _is_step(case):
        layer.capture()
    return layer


def run(state):
    case = state.case
    if case["kind"] == "qwen":
        out = {"logits": state.step()}
        if not _is_step(case):
            group = state.runner.cache.kv_groups[0]
            out.update(k=group.k, v=group.v)
        return out
    if state.graph is not None:
        state.graph.replay()
    else:
        for s in state.states:          # new sequences: their states start cleared
            s.zero_()
        state.once()
    out = {"rows": state.rows}
    out.update({f"state{i}": s for i, s in enumerate(state.states)})
    if case["kind"] in ("capped", "latent") and not _is_step(case):
        out["k"] = state.caches[0][1]
    return out


def tolerance(case):
    """About four times the errors against ``exact`` that were measured: 2.7e-6 in float32 (two layers and the head), 0.0017 to
    0.0028 for a bfloat16 layer, 0.008 for the logits of a bfloat16 model, whose roundings travel through its layers."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 0.03 if case["kind"] == "qwen" else 0.01}


def work(case):
    z, d, h = SIZES[case["size"]], _dims(case), SIZES[case["size"]]["hidden"]
    lens, starts = _lens(case), _starts(case)
    t, n = sum(lens), len(lens)
    e = 4 if case["dtype"] == "float32" else 2

    def pairs(window=None):     # (query, key) pairs that the mask lets see each other, and keys read
        total = sum(min(s + j + 1, window or 1 << 30) for s, m in zip(starts, lens) for j in range(m))
        return total, sum(min(s + m, (window or 1 << 30) + m - 1) for s, m in zip(starts, lens))

    kind = case["kind"]
    if kind == "qwen":
        nq, nk, inter = z["qwen_heads"] * 128, 1024, z["inter"]
        per = (nq + 2 * nk) * h + nq * h + 3 * h * inter
        seen, keys = pairs()
        return {"bytes": e * (case["layers"] * (per + 2 * 1024 * keys) + VOCAB * h + t * h) + 4 * n * VOCAB,
                "flops": case["layers"] * (2 * t * per + 4 * seen * nq) + 2 * n * VOCAB * h}
    rows = t * h * (e + 8)                  # activations in, residual read and written
    if kind == "moe":
        distinct = min(z["experts"], z["experts"] * (1 - (1 - z["top"] / z["experts"]) ** t))
        used = distinct * 3 * z["ff"] + 3 * z["shared"] + z["experts"]
        return {"bytes": int(e * h * used) + rows, "flops": 2 * t * h * (z["top"] * 3 * z["ff"] + 3 * z["shared"] + z["experts"])}
    if kind == "delta":
        weights, state, ops = h * (2 * d["nkv"] + 3 * d["nh"]) * 128 + 2 * d["nh"] * h, d["nh"] * 128 * 128, 6
    elif kind == "ssd":
        weights = h * (3 * d["ssd_heads"] * 64 + 2 * d["groups"] * 128 + d["ssd_heads"])
        state, ops = d["ssd_heads"] * 128 * 64, 4
    elif kind == "wkv":
        weights, state, ops = 5 * h * h + 128 * h, d["wkv_heads"] * 64 * 64, 4
    if kind in ("delta", "ssd", "wkv"):
        return {"bytes": e * weights + rows + 4 * n * state * (2 if _is_step(case) else 1), "flops": 2 * t * weights + ops * t * state}
    if kind == "capped":
        seen, keys = pairs(z["window"])
        nq, nk = z["heads"] * 128, z["heads"] // 4 * 128
        weights = h * (3 * nq + 2 * nk)
        return {"bytes": e * (weights + 2 * nk * keys) + rows, "flops": 2 * t * weights + 4 * seen * nq}
    seen, keys = pairs()
    nh, dim, rot, vd, rank = z["latent_heads"], z["latent_dim"], z["latent_rot"], z["latent_vdim"], z["rank"]
    weights = h * (nh * (dim + rot) + rank + rot + nh + nh * vd) + nh * (dim + vd) * rank
    per = 2 * (dim + rot + vd) if not _is_step(case) else 2 * (2 * rank + rot)
    return {"bytes": e * (weights + keys * (rank + rot)) + rows, "flops": 2 * t * weights + seen * nh * per}


# ---------------------------------------------------------------- the same in 64 bits, in plain torch

def _mm(x, w):
    return x @ w.double().T


def _rms(x):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + EPS)


def _cut(case, x):
    return torch.split(x, _lens(case))


def _conv(u, taps, past, bias=None):
    """(filtered rows, the last inputs) of one sequence; ``past`` [taps - 1, channels]."""
    k = taps.shape[1]
    if past is None:
        past = torch.zeros(k - 1, u.shape[1], dtype=u.dtype, device=DEV)
    x = torch.cat([past.double(), u])
    y = sum(x[j:j + u.shape[0]] * taps[:, j].double() for j in range(k))
    return (y if bias is None else y + bias.double()), x[x.shape[0] - (k - 1):]


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, pos, theta, pairs):
    """Rotation of the last axis of x [tokens, ..., dims]; the angle is a 32-bit product, as the design has it."""
    dims = x.shape[-1]
    f = (theta ** (-torch.arange(0, dims, 2, dtype=torch.float64) / dims)).to(torch.float32).to(DEV)
    a = (pos.to(torch.float32)[:, None] * f).double()
    a = a.view(a.shape[:1] + (1,) * (x.dim() - 2) + a.shape[1:])
    c, s = torch.cos(a), torch.sin(a)
    if pairs:
        p, q = x[..., 0::2], x[..., 1::2]
        return torch.stack([p * c - q * s, q * c + p * s], dim=-1).flatten(-2)
    p, q = x[..., :dims // 2], x[..., dims // 2:]
    return torch.cat([p * c - q * s, q * c + p * s], dim=-1)


def _attend(q, k, v, start, window=None, cap=0.0):
    """q [t, heads, d] over keys [n, kv heads, d] whose last t are the queries' own."""
    t, nh, n, nkv = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    own = torch.arange(n - t, n, device=DEV)[:, None]
    key = torch.arange(n, device=DEV)[None]
    hide = (key > own) if window is None else (key > own) | (key <= own - window)
    out = []
    for i in range(nkv):
        s = torch.einsum("tgd,nd->gtn", q[:, i * (nh // nkv):(i + 1) * (nh // nkv)], k[:, i])
        if cap:
            s = cap * torch.tanh(s / cap)
        out.append(torch.einsum("gtn,nd->tgd", torch.softmax(s.masked_fill(hide, -math.inf), -1), v[:, i]))
    return torch.cat(out, 1)


def _exact_scan(case, made):
    w, h, d = made["w"], made["h"].double(), _dims(case)
    past, kind = made["past"], case["kind"]
    ys, filters, states = [], [], []
    for i, x in enumerate(_cut(case, h)):
        t = x.shape[0]
        before = past["filter"][i] if past else None
        if kind == "delta":
            nh, rep, a, b = d["nh"], d["nh"] // d["nkv"], _mm(x, w["a"]), _mm(x, w["b"])
            f, last = _conv(torch.cat([_mm(x, w[s]) for s in "qkv"], 1), torch.cat([w[s + "_conv"] for s in "qkv"]), before)
            q, k, v = (s.view(t, -1, 128) for s in torch.split(_silu(f), [d["nkv"] * 128, d["nkv"] * 128, nh * 128], 1))
            q, k = (s / torch.sqrt(s.square().sum(-1, keepdim=True) + 1e-6) for s in (q, k))
            q, k = (s.repeat_interleave(rep, 1) for s in (q * 128 ** -0.5, k))
            g = torch.exp(-torch.exp(w["A_log"].double()) * torch.nn.functional.softplus(a + w["dt_bias"].double()))[..., None, None]
            beta, gate, norm = torch.sigmoid(b)[..., None], _silu(_mm(x, w["g"])).view(t, nh, 128), w["norm"].double()
        elif kind == "ssd":
            nh, inner, gn = d["ssd_heads"], d["ssd_heads"] * 64, d["groups"] * 128
            zz, u, dt = torch.split(_mm(x, w["in"]), [inner, inner + 2 * gn, nh], 1)
            f, last = _conv(u, w["conv"], before, w["conv_bias"])
            v, k, q = (s.view(t, -1, m) for s, m in zip(torch.split(_silu(f), [inner, gn, gn], 1), (64, 128, 128)))
            q, k = (s.repeat_interleave(nh // d["groups"], 1) for s in (q, k))
            dt = torch.nn.functional.softplus(dt + w["dt_bias"].double())
            g, k = torch.exp(-torch.exp(w["A_log"].double()) * dt)[..., None, None], k * dt[..., None]
        else:
            nh = d["wkv_heads"]
            was = torch.cat([before.double()[None] if before is not None else torch.zeros_like(x[:1]), x[:-1]])
            mix = {s: x + (was - x) * w["mu_" + s].double() for s in "rkvgw"}
            if case["dtype"] == "bfloat16":     # the blends are stored activations: rounded once, like h itself
                mix = {s: m.float().bfloat16().double() for s, m in mix.items()}
            q, k, v = (_mm(mix[s], w[s]).view(t, nh, 64) for s in "rkv")
            g = torch.exp(-torch.exp(w["w0"].double() + _mm(torch.tanh(_mm(mix["w"], w["w1"])), w["w2"]))).view(t, nh, 64, 1)
            gate, norm, last = _silu(_mm(mix["g"], w["g"])).view(t, nh, 64), w["norm"].double().view(nh, 64), x[-1]
        S = past["S"][i].double() if past else torch.zeros(nh, q.shape[-1], v.shape[-1], dtype=torch.float64, device=DEV)
        y = torch.empty_like(v)
        for j in range(t):
            if kind == "wkv":
                y[j] = torch.einsum("hd,hdv->hv", q[j], S) + (q[j] * w["u"].double() * k[j]).sum(-1, keepdim=True) * v[j]
                S = g[j] * S + k[j][:, :, None] * v[j][:, None]
                continue
            S = g[j] * S
            new = v[j] if kind == "ssd" else beta[j] * (v[j] - torch.einsum("hd,hdv->hv", k[j], S))
            S = S + k[j][:, :, None] * new[:, None]
            y[j] = torch.einsum("hd,hdv->hv", q[j], S)
        if kind == "ssd":
            y = (y + w["D"].double()[:, None] * v).reshape(t, -1) * _silu(zz)
            y = _rms(y.view(t, d["groups"], -1)).reshape(t, -1) * w["norm"].double()
        else:
            y = (_rms(y) * norm * gate).reshape(t, -1)
        ys.append(_mm(y, w["o"]))
        filters.append(last)
        states.append(_state_order(S[None])[0])
    return {"rows": made["x"].double() + torch.cat(ys), "state0": torch.stack(filters), "state1": torch.stack(states)}


def _exact_capped(case, made):
    w, z = made["w"], SIZES[case["size"]]
    nh, nk = z["heads"], z["heads"] // 4
    out, filters = [], []
    for i, x in enumerate(_cut(case, made["h"].double())):
        t, start = x.shape[0], _starts(case)[i]
        u = torch.cat([_mm(x, w[s]) + w[s + "_bias"].double() for s in "qkv"], 1)
        f, last = _conv(u, torch.cat([w[s + "_conv"] for s in "qkv"]), made["past"]["filter"][i] if made["past"] else None)
        q, k, v = (s.view(t, -1, 128) for s in torch.split(f, [nh * 128, nk * 128, nk * 128], 1))
        pos = torch.arange(start, start + t, device=DEV)
        q, k = _rotate(q, pos, 1e6, False) * 128 ** -0.5, _rotate(k, pos, 1e6, False)
        if made["past"]:
            k, v = torch.cat([made["past"]["k"][i].double(), k]), torch.cat([made["past"]["v"][i].double(), v])
        o = _attend(q, k, v, start, z["window"], 30.0).reshape(t, -1) * torch.sigmoid(_mm(x, w["g"]))
        out.append(_mm(o, w["o"]))
        filters.append(last)
    got = {"rows": made["x"].double() + torch.cat(out), "state0": torch.stack(filters)}
    return got if _is_step(case) else {**got, "k": None}


def _exact_latent(case, made):
    w, z = made["w"], SIZES[case["size"]]
    nh, dim, rot, vd, rank = z["latent_heads"], z["latent_dim"], z["latent_rot"], z["latent_vdim"], z["rank"]
    out = []
    for i, x in enumerate(_cut(case, made["h"].double())):
        t, start = x.shape[0], _starts(case)[i]
        pos = torch.arange(start, start + t, device=DEV)
        q = _mm(x, w["q"]).view(t, nh, dim + rot)
        kv = _mm(x, w["dkv"])
        rows = torch.cat([_rms(kv[:, :rank]) * w["dkv_norm"].double(), _rotate(kv[:, rank:], pos, 1e4, True)], 1)
        if made["past"]:
            rows = torch.cat([made["past"]["rows"][i].double(), rows])
        q = torch.cat([q[..., :dim], _rotate(q[..., dim:], pos, 1e4, True)], -1) * (dim + rot) ** -0.5
        o = []
        for a in range(nh):
            k = torch.cat([_mm(rows[:, :rank], w["uk"][a * dim:(a + 1) * dim]), rows[:, rank:]], 1)[:, None]
            v = _mm(rows[:, :rank], w["uv"][a * vd:(a + 1) * vd])[:, None]
            o.append(_attend(q[:, a:a + 1], k, v, start))
        o = torch.cat(o, 1) * torch.sigmoid(_mm(x, w["g"]))[..., None]
        out.append(_mm(o.reshape(t, -1), w["o"]))
    got = {"rows": made["x"].double() + torch.cat(out)}
    return got if _is_step(case) else {**got, "k": None}


def _exact_moe(case, made):
    w, z, h = made["w"], SIZES[case["size"]], made["h"].double()

    def act(gate, up):
        gate, up = gate.clamp(max=7.0), up.clamp(-7.0, 7.0)
        return gate * torch.sigmoid(1.702 * gate) * (up + 1.0)

    logits = _mm(h, w["router"]) + w["router_bias"].double()
    top, idx = torch.topk(logits, z["top"], dim=1)
    wts = torch.softmax(top, 1)
    out = torch.sigmoid(_mm(h, w["shared.sg"])) * _mm(act(_mm(h, w["shared.gate"]), _mm(h, w["shared.up"])), w["shared.down"])
    for e in range(z["experts"]):
        tok, slot = torch.nonzero(idx == e, as_tuple=True)
        if tok.numel():
            y = _mm(act(_mm(h[tok], w[f"e{e}.gate"]), _mm(h[tok], w[f"e{e}.up"])), w[f"e{e}.down"])
            out.index_add_(0, tok, y * wts[tok, slot][:, None])
    return {"rows": made["x"].double() + out}


def _exact_qwen(case, seed):
    w, ids, past = _qwen_made(case, seed)
    z = SIZES[case["size"]]
    xs = [w["model.embed_tokens.weight"][i].double() for i in _cut(case, ids)]
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        a = p + "self_attn."
        for i, x in enumerate(xs):
            t, start = x.shape[0], _starts(case)[i]
            pos = torch.arange(start, start + t, device=DEV)
            h = _rms(x) * w[p + "input_layernorm.weight"].double()
            q, k, v = (_mm(h, w[a + s + "_proj.weight"]).view(t, -1, 128) for s in "qkv")
            q = _rotate(_rms(q) * w[a + "q_norm.weight"].double(), pos, 1e6, False) * 128 ** -0.5
            k = _rotate(_rms(k) * w[a + "k_norm.weight"].double(), pos, 1e6, False)
            if start:
                k, v = (torch.cat([old.double(), new]) for old, new in zip(past[layer][i], (k, v)))
            x = x + _mm(_attend(q, k, v, start).reshape(t, -1), w[a + "o_proj.weight"])
            h = _rms(x) * w[p + "post_attention_layernorm.weight"].double()
            xs[i] = x + _mm(_silu(_mm(h, w[p + "mlp.gate_proj.weight"])) * _mm(h, w[p + "mlp.up_proj.weight"]),
                            w[p + "mlp.down_proj.weight"])
    last = torch.stack([x[-1] for x in xs])
    head = w.get("lm_head.weight", w["model.embed_tokens.weight"])
    last = _rms(last) * w["model.norm.weight"].double()
    out = {"logits": torch.cat([_mm(last, head[a:a + 16384]) for a in range(0, VOCAB, 16384)], 1)}
    return out if _is_step(case) else {**out, "k": None, "v": None}


def exact(case, seed):
    if case["kind"] == "qwen":
        return _exact_qwen(case, seed)
    made = _made(case, seed)
    return {"capped": _exact_capped, "latent": _exact_latent, "moe": _exact_moe}.get(case["kind"], _exact_scan)(case, made)
