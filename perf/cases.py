"""The work that users of this engine have it do, as cases that can be timed and compared.

Four kinds, each through the calls a program makes:

  steps       a whole Qwen3 model through ``ModelRunner.step``: the prompts of all requests as one step, then one given
              token per request and step (what trace replay does, and generation with the sampler left out)
  attention   one attention layer (projections, norm, rotation, cache write, attention, output product) through the
              part's ``forward``: prompt portions, with or without keys of earlier steps, and single tokens
  recurrence  the layers with a state per request through ``ops``: delta rule, constant decays, state space
  experts     a mixture of experts with its shared unit through the part's ``forward``

Sizes are those of ``bench.py`` (Qwen3-8B and Qwen3-0.6B, and the ``8b`` and ``1b`` sizes of its design benches) and odd
ones around them.  Inputs, weights and the keys of earlier steps come from the seed alone.
"""
from __future__ import annotations

import math

import torch

from tiny_llm_infer_b200 import ops
from tiny_llm_infer_b200.cache import CacheManager
from tiny_llm_infer_b200.config.base import describe_model
from tiny_llm_infer_b200.config.qwen3 import Qwen3Config
from tiny_llm_infer_b200.engine import ModelRunner, StepEntry
from tiny_llm_infer_b200.engine.batch import StepContext
from tiny_llm_infer_b200.engine.runner import strict_float32
from tiny_llm_infer_b200.models.model import Model
from tiny_llm_infer_b200.parts import PartSpec, lookup

DEV = "cuda:0"
PAGE = 16
TYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# --------------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest call: one chat request on the smallest model; launches and latency are all of it
        dict(name="steps_one_request", kind="steps", width=1024, ff=3072, layers=28, heads=16, kv_heads=8, dim=128,
             vocab=151936, requests=1, prompt=16, steps=8),
        # eight requests of 128 tokens and some generation, at the width of the 8B model
        dict(name="steps_eight_requests", kind="steps", width=4096, ff=12288, layers=4, heads=32, kv_heads=8, dim=128,
             vocab=32768, requests=8, prompt=128, steps=16),
        # a prompt through an attention with cap, window, learned sink and a gate per head (Sozavik, Panolorn, Vigonex)
        dict(name="attention_capped_prompt", kind="attention", style="capped", dtype="bfloat16", width=4096, heads=32,
             kv_heads=8, dim=128, requests=1, tokens=2048, before=0, window=4096),
        # a late portion of a long prompt through Qwen3's attention, of an odd length
        dict(name="attention_plain_portion", kind="attention", style="plain", dtype="bfloat16", width=4096, heads=32,
             kv_heads=8, dim=128, requests=1, tokens=509, before=3587, window=0),
        # sixty-four requests that each decode a token at contexts around 2000
        dict(name="attention_capped_single", kind="attention", style="capped", dtype="bfloat16", width=4096, heads=32,
             kv_heads=8, dim=128, requests=64, tokens=1, before=2000, window=4096),
        # the true float32 path (replay against recorded logits) on two prompts
        dict(name="attention_plain_float32", kind="attention", style="plain", dtype="float32", width=1024, heads=16,
             kv_heads=8, dim=128, requests=2, tokens=300, before=0, window=0),
        # a prompt through the delta rule with a decay per channel (Kaketar; Tetodra and Vigonex have relatives)
        dict(name="recurrence_delta_prompt", kind="recurrence", rule="delta", heads=32, kv_heads=32, dk=128, dv=128,
             requests=1, tokens=2048),
        # three prompts through the recurrence with constant decays (Sozavik)
        dict(name="recurrence_fixed_prompts", kind="recurrence", rule="fixed", heads=32, kv_heads=32, dk=128, dv=128,
             requests=3, tokens=701),
        # a prompt portion of an odd length through the state space (Pevolorn)
        dict(name="recurrence_space_prompt", kind="recurrence", rule="space", heads=64, kv_heads=8, dk=128, dv=64,
             requests=1, tokens=1023),
        # sixty-four requests that each decode a token through the delta rule
        dict(name="recurrence_delta_single", kind="recurrence", rule="delta", heads=32, kv_heads=32, dk=128, dv=128,
             requests=64, tokens=1),
        # a mixture of experts when eight requests decode
        dict(name="experts_eight_rows", kind="experts", width=4096, experts=64, top=4, ff=2048, shared=4096, rows=8),
        # the same in a prompt of 2048 tokens
        dict(name="experts_prompt", kind="experts", width=4096, experts=64, top=4, ff=2048, shared=4096, rows=2048),
    ]


def _between(rng, lo, hi):
    """A whole number whose logarithm is spread evenly."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["steps", "attention", "attention", "recurrence", "recurrence", "experts"])
    if kind == "steps":
        width = rng.choice([1024, 2048, 4096])
        kv_heads = rng.choice([4, 8])
        return dict(kind=kind, width=width, ff=3 * width, layers=rng.randint(2, 4), heads=kv_heads * rng.choice([2, 4]),
                    kv_heads=kv_heads, dim=128, vocab=32768, requests=_between(rng, 1, 8), prompt=_between(rng, 16, 128),
                    steps=rng.randint(4, 16))
    if kind == "attention":
        style, single = rng.choice(["capped", "plain"]), rng.random() < 0.4
        kv_heads, wide = rng.choice([4, 8]), rng.random() < 0.5
        dtype = "float32" if style == "plain" and rng.random() < 0.3 else "bfloat16"
        requests = _between(rng, 4, 64) if single else rng.randint(1, 3)
        most = (300 if dtype == "float32" else 2048) // requests
        return dict(kind=kind, style=style, dtype=dtype, width=4096 if wide else 2048, heads=kv_heads * (4 if wide else 2),
                    kv_heads=kv_heads, dim=128, requests=requests, tokens=1 if single else _between(rng, 64, most),
                    before=_between(rng, 64, 2000) if single else rng.choice([0, 0, _between(rng, 16, 1500)]),
                    window=4096 if style == "capped" else 0)
    if kind == "recurrence":
        rule, single = rng.choice(["delta", "fixed", "space"]), rng.random() < 0.35
        requests = _between(rng, 1, 64) if single else rng.randint(1, 8)
        heads = rng.choice([16, 32])
        tokens = 1 if single else _between(rng, 64, 2048 // requests)
        if rule == "space":
            return dict(kind=kind, rule=rule, heads=2 * heads, kv_heads=8, dk=rng.choice([64, 128]), dv=64,
                        requests=requests, tokens=tokens)
        dk = rng.choice([64, 128])
        return dict(kind=kind, rule=rule, heads=heads, kv_heads=heads, dk=dk, dv=128, requests=requests, tokens=tokens)
    wide = rng.random() < 0.5
    return dict(kind=kind, width=4096 if wide else 2048, experts=64 if wide else 32, top=4, ff=2048 if wide else 1024,
                shared=4096 if wide else 2048, rows=_between(rng, 1, 2048))


# --------------------------------------------------------------------------- inputs
class _Draws:
    """Tensors from one generator on the device, in the order they are asked for."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=dtype, device=DEV)
        return t.normal_(mean, std, generator=self.gen)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        t = torch.empty(shape, dtype=dtype, device=DEV)
        return t.uniform_(lo, hi, generator=self.gen)

    def ints(self, top, n):
        return torch.randint(0, top, (n,), generator=self.gen, device=DEV)


def _lengths(case):
    """Tokens of every request of a step: the first has all, the others fall short of it by a little more each."""
    n = case["tokens"] if case["kind"] != "steps" else case["prompt"]
    return [max(1, n - (5 * r) % max(1, n // 2)) for r in range(case["requests"])]


def _befores(case):
    return [max(0, case["before"] - (37 * r) % max(1, case["before"] // 2)) for r in range(case["requests"])]


def _steps_inputs(case, seed):
    d = _Draws(seed)
    bf, W, D, H, G = torch.bfloat16, case["width"], case["dim"], case["heads"], case["kv_heads"]
    w = {"model.embed_tokens.weight": d.normal(case["vocab"], W, std=0.02, dtype=bf)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w[p + "input_layernorm.weight"] = d.uniform(W, lo=0.8, hi=1.2, dtype=bf)
        w[p + "post_attention_layernorm.weight"] = d.uniform(W, lo=0.8, hi=1.2, dtype=bf)
        for name, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
            w[p + f"self_attn.{name}_proj.weight"] = d.normal(rows, W, std=0.02, dtype=bf)
        w[p + "self_attn.o_proj.weight"] = d.normal(W, H * D, std=0.02, dtype=bf)
        for name in "qk":
            w[p + f"self_attn.{name}_norm.weight"] = d.uniform(D, lo=0.8, hi=1.2, dtype=bf)
        w[p + "mlp.gate_proj.weight"] = d.normal(case["ff"], W, std=0.02, dtype=bf)
        w[p + "mlp.up_proj.weight"] = d.normal(case["ff"], W, std=0.02, dtype=bf)
        w[p + "mlp.down_proj.weight"] = d.normal(W, case["ff"], std=0.02, dtype=bf)
    w["model.norm.weight"] = d.uniform(W, lo=0.8, hi=1.2, dtype=bf)
    w["lm_head.weight"] = d.normal(case["vocab"], W, std=0.02, dtype=bf)
    tokens = [d.ints(case["vocab"], n + case["steps"]).tolist() for n in _lengths(case)]
    return w, tokens


def _attention_inputs(case, seed):
    d = _Draws(seed)
    dt, W, D, H, G = TYPES[case["dtype"]], case["width"], case["dim"], case["heads"], case["kv_heads"]
    x = d.normal(sum(_lengths(case)), W, dtype=dt)
    if case["style"] == "plain":
        w = {f"{n}_proj.weight": d.normal(rows, W, std=0.02, dtype=dt) for n, rows in (("q", H * D), ("k", G * D), ("v", G * D))}
        w["o_proj.weight"] = d.normal(W, H * D, std=0.02, dtype=dt)
        w["q_norm.weight"], w["k_norm.weight"] = d.uniform(D, lo=0.8, hi=1.2, dtype=dt), d.uniform(D, lo=0.8, hi=1.2, dtype=dt)
    else:
        w = {n: d.normal(rows, W, std=0.02, dtype=dt) for n, rows in (("q", H * D), ("k", G * D), ("v", G * D), ("g", H))}
        w["o"] = d.normal(W, H * D, std=0.02, dtype=dt)
        w["sink"] = d.normal(H)
    old = [(d.normal(n, G, D, dtype=dt), d.normal(n, G, D, dtype=dt)) for n in _befores(case)]     # normed keys, values
    return x, w, old


def _lanes(dk):
    """Lanes over which the state's layout deals the dk rows of a column."""
    r = 4
    while r < 32 and -(-dk // r) > 16:
        r *= 2
    return r


def _pack_state(S):
    """[.., heads, dk, dv] in the layout of a request's state: row i = r * per + il lies at [il][column][r]."""
    *lead, heads, dk, dv = S.shape
    R = _lanes(dk)
    per = -(-dk // R)
    S = torch.nn.functional.pad(S, (0, 0, 0, R * per - dk))
    S = S.reshape(*lead, heads, R, per, dv).movedim(-3, -1)                     # [.., heads, per, dv, R]
    return S.reshape(*lead, heads * per * dv * R)


def _recurrence_inputs(case, seed):
    d = _Draws(seed)
    bf, rule, H, G, dk, dv = torch.bfloat16, case["rule"], case["heads"], case["kv_heads"], case["dk"], case["dv"]
    T, n = sum(_lengths(case)), case["requests"]
    t = {"S": d.normal(n, H, dk, dv, std=0.1)}
    if rule == "fixed":
        t["proj"] = d.normal(T, H * (2 * dk + 2 * dv), dtype=bf)
        t["decay"] = torch.exp(-torch.pow(2.0, -8.0 * torch.arange(1, H + 1, device=DEV, dtype=torch.float32) / H))
        t["out_weight"] = d.uniform(H * dv, lo=0.8, hi=1.2)
        return t
    channels = 2 * G * dk + H * dv
    t["conv_w"] = d.normal(channels, 4, std=0.5, dtype=bf)
    t["tail"] = d.normal(n, 3, channels)
    if rule == "delta":
        t["proj"] = d.normal(T, channels + H, dtype=bf)
        t["gate"] = d.normal(T, H * dv, dtype=bf)
        t["a"] = d.normal(T, H * dk)
        t["dt_bias"] = d.normal(H * dk, mean=-1.0)
        t["rate"] = torch.exp(d.uniform(H, lo=-4.0, hi=0.0))
        t["out_weight"] = d.uniform(dv, lo=0.8, hi=1.2)
    else:
        t["proj"] = d.normal(T, 2 * H * dv + 2 * G * dk + H, dtype=bf)
        t["conv_b"] = d.normal(channels, std=0.1)
        t["dt_bias"] = d.normal(H, mean=-2.0)
        t["rate"] = torch.exp(d.uniform(H, lo=0.0, hi=2.7))
        t["skip"] = d.uniform(H, lo=0.8, hi=1.2)
        t["out_weight"] = d.uniform(H * dv, lo=0.8, hi=1.2)
    return t


def _experts_inputs(case, seed):
    d = _Draws(seed)
    bf, W, F, E = torch.bfloat16, case["width"], case["ff"], case["experts"]
    x = d.normal(case["rows"], W, dtype=bf)
    w = {"router": d.normal(E, W, std=0.02, dtype=bf)}
    gate, up, down = d.normal(E, F, W, std=0.02, dtype=bf), d.normal(E, F, W, std=0.02, dtype=bf), d.normal(E, W, F, std=0.02, dtype=bf)
    for e in range(E):
        w[f"e{e}.gate"], w[f"e{e}.up"], w[f"e{e}.down"] = gate[e], up[e], down[e]
    for name, shape in (("gate", (case["shared"], W)), ("up", (case["shared"], W)), ("down", (W, case["shared"]))):
        w["s." + name] = d.normal(*shape, std=0.02, dtype=bf)
    return x, w


# --------------------------------------------------------------------------- what a program has in hand
def _int(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _context(slots, lengths, befores):
    """The step's context as the runner lays it out."""
    seg, tiles, dec, row = [], [], [], 0
    for s, (slot, n, p0) in enumerate(zip(slots, lengths, befores)):
        seg.append([slot, row, n, p0])
        if n == 1:
            dec.append(row)
        else:
            tiles += [(s, off, p0 + min(off + 64, n)) for off in range(0, n, 64)]
        row += n
    tiles.sort(key=lambda t: (t[1] % 256 != 0, t[1] % 128 != 0, -t[2]))
    return StepContext(
        tokens=row, token_ids=None, positions=_int([p0 + i for _, _, n, p0 in seg for i in range(n)]),
        token_slot=_int([slot for slot, _, n, _ in seg for _ in range(n)]), want_rows=None, segments=[], seg_info=_int(seg),
        dec_rows=None if len(dec) == row else _int(dec), n_dec=len(dec), pf_tiles=_int([t[:2] for t in tiles]).view(-1, 2),
        n_tiles=len(tiles), n_tiles128=sum(1 for t in tiles if t[1] % 128 == 0),
        n_tiles256=sum(1 for t in tiles if t[1] % 256 == 0), max_context=max(n + p0 for _, _, n, p0 in seg),
        max_segment=max(lengths))


def _mixer(case):
    H, G, D, W = case["heads"], case["kv_heads"], case["dim"], case["width"]
    dt = TYPES[case["dtype"]]
    if case["style"] == "plain":
        return lookup("mixer", "gq_attention")(W, H, G, D, dt, DEV, qk_norm_eps=1e-6,
                                               position=PartSpec("rotary_half", {"head_dim": D, "theta": 1e6}))
    return lookup("mixer", "biased_attention")(W, H, G, D, D, D ** -0.5, dt, DEV, unit_norm_eps=1e-6, softcap=50.0,
                                               window=case["window"], sink=True, learned_sink=True, output_gate=True,
                                               gate_per_head=True)


def prepare(case, seed):
    strict_float32()
    if case["kind"] == "steps":
        w, tokens = _steps_inputs(case, seed)
        cfg = Qwen3Config(hidden_size=case["width"], intermediate_size=case["ff"], num_hidden_layers=case["layers"],
                          num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=case["dim"],
                          vocab_size=case["vocab"], max_position_embeddings=4096, tie_word_embeddings=False,
                          layer_types=("full_attention",) * case["layers"])
        model = Model(describe_model(cfg), torch.bfloat16, DEV)
        model.load(w)
        longest = case["prompt"] + case["steps"]
        cache = CacheManager(model.cache_needs(), PAGE, case["requests"] * (-(-longest // PAGE) + 1), max_slots=case["requests"],
                             max_seq_len=longest, dtype=torch.bfloat16, device=DEV)
        return dict(kind="steps", runner=ModelRunner(model, cache, max_batch_tokens=max(64, sum(_lengths(case)))), tokens=tokens,
                    prompts=_lengths(case), steps=case["steps"])
    if case["kind"] == "attention":
        x, w, old = _attention_inputs(case, seed)
        mixer = _mixer(case)
        mixer.load(w)
        lengths, befores = _lengths(case), _befores(case)
        longest = max(n + p for n, p in zip(lengths, befores))
        cache = CacheManager({0: (mixer.cache_spec(), None)}, PAGE, len(lengths) * -(-longest // PAGE), max_slots=len(lengths),
                             max_seq_len=longest, dtype=TYPES[case["dtype"]], device=DEV)
        for r, (n, p0) in enumerate(zip(lengths, befores)):
            cache.admit(r)
            cache.reserve(r, n + p0)
        cache.sync()
        view = cache.view(0)
        for r, (k, v) in enumerate(old):
            n = k.shape[0]
            pages = view.block_table[cache.slot_of(r)].long()
            at = torch.arange(n, device=DEV)
            for plane, rows in zip(view.planes, (k, v)):
                plane[pages[at // PAGE], :, at % PAGE] = rows
        ctx = _context([cache.slot_of(r) for r in range(len(lengths))], lengths, befores)
        return dict(kind="attention", mixer=mixer, x=x, ctx=ctx, view=view)
    if case["kind"] == "recurrence":
        t = _recurrence_inputs(case, seed)
        state = _pack_state(t["S"])
        if "tail" in t:
            state = torch.cat([state, t["tail"].flatten(1)], dim=1)
            t["conv_t"] = t["conv_w"].t().contiguous()
        lengths = _lengths(case)
        ctx = _context(range(len(lengths)), lengths, [0] * len(lengths))
        return dict(t, kind="recurrence", case=case, state=state.contiguous(), token_slot=ctx.token_slot,
                    seg_info=None if case["tokens"] == 1 else ctx.seg_info)
    x, w = _experts_inputs(case, seed)
    part = lookup("feed_forward", "moe")(case["width"], case["experts"], case["top"], case["ff"], torch.bfloat16, DEV,
                                         shared=PartSpec("swiglu", dict(hidden_size=case["width"], intermediate_size=case["shared"],
                                                                        names=("gate", "up", "down")), prefix="s."))
    part.load(w)
    return dict(kind="experts", part=part, x=x)


# --------------------------------------------------------------------------- one pass
@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "steps":
        runner, prompts, out = state["runner"], state["prompts"], []
        entries = [StepEntry(r, toks[:n], [n - 1]) for r, (toks, n) in enumerate(zip(state["tokens"], prompts))]
        out.append(runner.step(entries).clone())
        for i in range(state["steps"]):
            entries = [StepEntry(r, [toks[n + i]], [0]) for r, (toks, n) in enumerate(zip(state["tokens"], prompts))]
            out.append(runner.step(entries).clone())
        for r in range(len(prompts)):
            runner.release(r)
        return out
    if kind == "attention":
        state["ctx"].memo.clear()
        y = state["mixer"].forward(state["x"], state["ctx"], state["view"])
        return {"y": y, "keys": state["view"].planes[0], "values": state["view"].planes[1]}
    if kind == "experts":
        return state["part"].forward(state["x"], None)
    c, t, bf = state["case"], state, torch.bfloat16
    H, G, dk, dv = c["heads"], c["kv_heads"], c["dk"], c["dv"]
    if c["rule"] == "fixed":
        y = ops.linear_recurrence(t["proj"], "fixed_decay", None, t["decay"], 1.0, t["proj"][:, H * (2 * dk + dv):], "sigmoid",
                                  t["out_weight"], True, 1e-6, t["token_slot"], t["seg_info"], t["state"], H, dk, dv, 1.0, bf,
                                  input_act="silu", norm_whole=True)
    elif c["rule"] == "delta":
        y = ops.delta_rule(t["proj"], t["conv_w"], 4, t["a"], t["dt_bias"], t["rate"], t["gate"], t["out_weight"], 1e-6,
                           t["token_slot"], t["seg_info"], t["state"], H, G, dk, dv, dk ** -0.5, 1e-6, bf, conv_t=t["conv_t"])
    else:
        y = ops.state_space(t["proj"], t["conv_w"], t["conv_b"], 4, t["dt_bias"], t["rate"], t["skip"], t["out_weight"], 1e-6, G,
                            t["token_slot"], t["seg_info"], t["state"], H, G, dk, dv, bf, conv_t=t["conv_t"])
    return {"y": y, "state": t["state"]}


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    if case["kind"] == "steps":
        W, D, H, G, n = case["width"], case["dim"], case["heads"], case["kv_heads"], _lengths(case)
        layer = W * (H + 2 * G) * D + H * D * W + 3 * W * case["ff"]
        head, rows, T = W * case["vocab"], case["requests"], sum(n)
        pairs = sum(m * (m + 1) / 2 for m in n) + case["steps"] * sum(m + case["steps"] / 2 for m in n)
        reads = sum(case["steps"] * (m + case["steps"] / 2) for m in n)
        return {"bytes": 2.0 * (case["steps"] + 1) * (case["layers"] * layer + head) + case["layers"] * 4.0 * G * D * (T + reads)
                + 4.0 * rows * (case["steps"] + 1) * case["vocab"],
                "flops": 2.0 * case["layers"] * layer * (T + rows * case["steps"]) + 2.0 * head * rows * (case["steps"] + 1)
                + 4.0 * case["layers"] * H * D * pairs}
    if case["kind"] == "attention":
        W, D, H, G, n, p = case["width"], case["dim"], case["heads"], case["kv_heads"], _lengths(case), _befores(case)
        size, T = 4 if case["dtype"] == "float32" else 2, sum(n)
        weights = W * (H + 2 * G) * D + H * D * W + (H * W if case["style"] == "capped" else 0)
        pairs = sum(m * b + m * (m + 1) / 2 for m, b in zip(n, p))
        return {"bytes": size * (weights + 2.0 * T * W + 2.0 * G * D * (T + sum(p))), "flops": 2.0 * T * weights + 4.0 * H * D * pairs}
    if case["kind"] == "experts":
        W, F, S, T = case["width"], case["ff"], case["shared"], case["rows"]
        E = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** T)          # experts that some row chooses
        return {"bytes": 2.0 * (3 * E * F * W + 3 * S * W + case["experts"] * W + 2 * T * W),
                "flops": 2.0 * T * (3 * case["top"] * F * W + 3 * S * W + case["experts"] * W)}
    H, G, dk, dv, T, n = case["heads"], case["kv_heads"], case["dk"], case["dv"], sum(_lengths(case)), case["requests"]
    columns = {"delta": 2 * (2 * G * dk + 3 * H * dv + H) + 4 * H * dk, "fixed": 2 * (2 * H * dk + 3 * H * dv),
               "space": 2 * (3 * H * dv + 2 * G * dk + H)}[case["rule"]]
    return {"bytes": 8.0 * n * H * dk * dv + 1.0 * T * columns, "flops": T * H * dk * dv * (7.0 if case["rule"] == "delta" else 5.0)}


def tolerance(case):
    # measured against exact() (2-norm of the difference over that of the result), and about four times that
    if case["kind"] == "steps":
        return {"rel": 0.03, "max": 0.2}              # 0.8% (28 layers of width 1024), 1.4% (4 layers of width 4096)
    if case["kind"] == "attention":
        if case["dtype"] == "float32":
            return {"rel": 1e-5, "max": 1e-4}         # 0.00012%; sums of up to 2048 float32 products in any order
        return {"rel": 0.015, "max": 0.2}             # 0.35 to 0.44%: projections, queries, keys and heads in bfloat16
    if case["kind"] == "recurrence":
        return {"rel": 0.007, "max": 0.1}             # 0.17%: the result's own rounding to bfloat16
    return {"rel": 0.013, "max": 0.2}                 # 0.33%: the experts' hidden rows and the result in bfloat16


# --------------------------------------------------------------------------- the same in 64 bits
def _norm(x, eps, gain=None):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if gain is None else y * gain.double()


def _rotate(x, pos, theta=1e6):
    """[T, heads, D]: element i turns with element i + D / 2."""
    half = x.shape[-1] // 2
    freq = (theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)).float()
    angle = (pos.float()[:, None] * freq[None, :]).double()[:, None]
    a, b, c, s = x[..., :half], x[..., half:], angle.cos(), angle.sin()
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _attend(q, k, v, p0, scale, cap=0.0, window=0, sink=None):
    """q [T, H, D] at positions p0 .. over k, v [p0 + T, G, D]."""
    T, H, D = q.shape
    n, G, _ = k.shape
    i, j = torch.arange(p0, p0 + T, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
    hidden = (j > i) | ((i - j >= window) if window else torch.zeros((), dtype=torch.bool, device=q.device))
    out = torch.empty_like(q)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].t()) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(T, 1)], 1)
        out[:, h] = torch.softmax(s, 1)[:, :n] @ v[:, h * G // H]
    return out


def _mm(x, w):
    return x @ w.double().t()


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "steps":
        return _exact_steps(case, seed)
    if case["kind"] == "attention":
        return _exact_attention(case, seed)
    if case["kind"] == "experts":
        return _exact_experts(case, seed)
    return _exact_recurrence(case, seed)


def _exact_steps(case, seed):
    w, tokens = _steps_inputs(case, seed)
    H, G, D, lengths = case["heads"], case["kv_heads"], case["dim"], _lengths(case)
    rows = []
    for toks, n in zip(tokens, lengths):
        pos = torch.arange(len(toks), device=DEV)
        h = w["model.embed_tokens.weight"][torch.tensor(toks, device=DEV)].double()
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            x = _norm(h, 1e-6, w[p + "input_layernorm.weight"])
            q, k, v = (_mm(x, w[p + f"self_attn.{m}_proj.weight"]).view(len(toks), -1, D) for m in "qkv")
            q = _rotate(_norm(q, 1e-6, w[p + "self_attn.q_norm.weight"]), pos)
            k = _rotate(_norm(k, 1e-6, w[p + "self_attn.k_norm.weight"]), pos)
            h = h + _mm(_attend(q, k, v, 0, D ** -0.5).flatten(1), w[p + "self_attn.o_proj.weight"])
            x = _norm(h, 1e-6, w[p + "post_attention_layernorm.weight"])
            x = torch.nn.functional.silu(_mm(x, w[p + "mlp.gate_proj.weight"])) * _mm(x, w[p + "mlp.up_proj.weight"])
            h = h + _mm(x, w[p + "mlp.down_proj.weight"])
        rows.append(_mm(_norm(h[n - 1:n + case["steps"]], 1e-6, w["model.norm.weight"]), w["lm_head.weight"]))
    return [torch.stack([r[i] for r in rows]) for i in range(case["steps"] + 1)]


def _exact_attention(case, seed):
    x, w, old = _attention_inputs(case, seed)
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    plain, out, row = case["style"] == "plain", [], 0
    for n, p0, (k_old, v_old) in zip(_lengths(case), _befores(case), old):
        xr = x[row:row + n].double()
        row += n
        q, k, v = (_mm(xr, w[m + ("_proj.weight" if plain else "")]).view(n, -1, D) for m in "qkv")
        q, k = _norm(q, 1e-6, w["q_norm.weight"] if plain else None), _norm(k, 1e-6, w["k_norm.weight"] if plain else None)
        if plain:
            pos = torch.arange(p0, p0 + n, device=DEV)
            q, k = _rotate(q, pos), _rotate(k, pos)
        k, v = torch.cat([k_old.double(), k]), torch.cat([v_old.double(), v])
        if plain:
            o = _attend(q, k, v, p0, D ** -0.5)
        else:
            o = _attend(q, k, v, p0, D ** -0.5, 50.0, case["window"], w["sink"]) * torch.sigmoid(_mm(xr, w["g"]))[..., None]
        out.append(_mm(o.flatten(1), w["o_proj.weight" if plain else "o"]))
    return {"y": torch.cat(out), "keys": None, "values": None}


def _exact_experts(case, seed):
    x, w = _experts_inputs(case, seed)
    x = x.double()

    def unit(u, p):
        return _mm(torch.nn.functional.silu(_mm(u, w[p + "gate"])) * _mm(u, w[p + "up"]), w[p + "down"])
    z = _mm(x, w["router"])
    chosen = torch.zeros_like(z, dtype=torch.bool).scatter_(1, z.topk(case["top"], dim=1).indices, True)
    out = unit(x, "s.")
    for e in range(case["experts"]):
        rows = chosen[:, e].nonzero()[:, 0]
        if rows.numel():
            out[rows] += unit(torch.sigmoid(z[rows, e])[:, None] * x[rows], f"e{e}.")
    return out


def _exact_recurrence(case, seed):
    t = _recurrence_inputs(case, seed)
    rule, H, G, dk, dv = case["rule"], case["heads"], case["kv_heads"], case["dk"], case["dv"]
    silu, sigmoid, softplus = torch.nn.functional.silu, torch.sigmoid, torch.nn.functional.softplus
    lengths = _lengths(case)
    proj, n_req, longest, row = t["proj"].double(), len(lengths), max(lengths), 0
    rows, inputs, tails = [], [], []
    first, channels = (H * dv if rule == "space" else 0), 2 * G * dk + H * dv
    for r, n in enumerate(lengths):
        rows.append(slice(row, row + n))
        row += n
        if rule == "fixed":
            inputs.append(silu(proj[rows[r], :2 * H * dk + H * dv]))
            continue
        c = torch.cat([t["tail"][r].double(), proj[rows[r], first:first + channels]])
        tails.append(c[-3:])
        y = sum(c[i:i + n] * t["conv_w"][:, i].double() for i in range(4))
        inputs.append(silu(y + t["conv_b"].double() if rule == "space" else y))
    xs = torch.zeros(n_req, longest, inputs[0].shape[1], dtype=torch.float64, device=DEV)
    for r, v in enumerate(inputs):
        xs[r, :lengths[r]] = v

    def spread(v, fill):                                    # [T, ...] to [requests, longest, ...]
        o = torch.full((n_req, longest) + tuple(v.shape[1:]), fill, dtype=torch.float64, device=DEV)
        for r in range(n_req):
            o[r, :lengths[r]] = v[rows[r]]
        return o
    if rule == "space":
        v, k, q = xs[..., :H * dv], xs[..., H * dv:H * dv + G * dk], xs[..., H * dv + G * dk:]
        dt = softplus(proj[:, 2 * H * dv + 2 * G * dk:] + t["dt_bias"].double())
        g = spread(torch.exp(-t["rate"].double() * dt), 1.0)[..., None]
        write = spread(dt, 0.0)
    else:
        q, k, v = xs[..., :G * dk], xs[..., G * dk:2 * G * dk], xs[..., 2 * G * dk:]
        write = torch.zeros(n_req, longest, H, dtype=torch.float64, device=DEV)
        for r in range(n_req):
            write[r, :lengths[r]] = 1.0
    q, k, v = (m.reshape(n_req, longest, -1, d) for m, d in ((q, dk), (k, dk), (v, dv)))
    if rule == "delta":
        q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
        k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        a = t["a"].double() + t["dt_bias"].double()
        g = spread(torch.exp(-t["rate"].double()[:, None] * softplus(a).view(-1, H, dk)), 1.0)
        write = spread(sigmoid(proj[:, channels:channels + H]), 0.0)
    elif rule == "fixed":
        g = torch.ones(n_req, longest, H, 1, dtype=torch.float64, device=DEV)
        for r in range(n_req):
            g[r, :lengths[r]] = t["decay"].double()[:, None]
    q, k = (m.repeat_interleave(H // m.shape[2], dim=2) for m in (q, k))
    S = t["S"].double()
    o = torch.empty(n_req, longest, H, dv, dtype=torch.float64, device=DEV)
    for i in range(longest):
        S = S * g[:, i, :, :, None]
        u = v[:, i] - torch.einsum("rhkv,rhk->rhv", S, k[:, i]) if rule == "delta" else v[:, i]
        S = S + k[:, i, :, :, None] * (write[:, i, :, None] * u)[:, :, None]
        o[:, i] = torch.einsum("rhkv,rhk->rhv", S, q[:, i])
    o = torch.cat([o[r, :lengths[r]] for r in range(n_req)])
    weight = t["out_weight"].double()
    if rule == "fixed":
        y = _norm(o.flatten(1), 1e-6) * weight * sigmoid(proj[:, H * (2 * dk + dv):])
        return {"y": y, "state": _pack_state(S)}
    if rule == "delta":
        y = (_norm(o, 1e-6) * weight).flatten(1) * sigmoid(t["gate"].double())
    else:
        skip = torch.cat([v[r, :lengths[r]] for r in range(n_req)]) * t["skip"].double()[:, None]
        y = (o + skip).flatten(1) * silu(proj[:, :H * dv])
        y = _norm(y.view(y.shape[0], G, -1), 1e-6).flatten(1) * weight
    return {"y": y, "state": torch.cat([_pack_state(S), torch.stack(tails).flatten(1)], dim=1)}
