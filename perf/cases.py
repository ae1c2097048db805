"""The work the framework is measured at: what a program that serves models with it has it do.

Two kinds of case. A `turn` is a whole call: an engine admits requests, runs their prompts in one
step and decodes given tokens one step at a time, reading logits each time. Every other kind is one
layer's part, made through the registry from a spec and called as a model calls it
(`part.forward(rows, step, cache)`): over the prompt portions of a few requests, or over single
tokens of many. Sizes are those of bench.py (the 8B shape; width 2048 and 4096 with its heads,
windows, states and experts) and generic ones around them.

Inputs and weights come from the seed alone; `exact` states each computation in plain torch in 64
bits from the same inputs.
"""
import math

import torch

from tgo_b200.config.spec import FeedForwardSpec, LayerSpec, MixerSpec, NormSpec, PositionSpec
from tgo_b200.engine.step import StepEntry
from tgo_b200.parts.base import LayerCache, StepContext
from tgo_b200.registry import BLOCKS, FEED_FORWARDS, MIXERS, NORMS

DEV = "cuda:0"
PAGE = 16
EPS = 1e-6
THETA = 5e5
BF = torch.bfloat16


def listed():
    return [
        # a single user's short exchange with a small dense model: launches and latency
        dict(name="turn_single", kind="turn", width=2048, heads=16, kv_heads=4, dim=128, ff=6144,
             layers=4, vocab=32768, requests=1, tokens=33, spread=0.0, steps=24),
        # a serving batch of the 8B shape: prompts of unlike lengths, then decoding together
        dict(name="turn_batch", kind="turn", width=4096, heads=32, kv_heads=8, dim=128, ff=12288,
             layers=2, vocab=32768, requests=24, tokens=301, spread=0.6, steps=24),
        # a prompt through one layer of the 8B shape
        dict(name="block_prompt", kind="block", dtype="bfloat16", width=4096, heads=32, kv_heads=8,
             dim=128, ff=12288, requests=1, tokens=2048, spread=0.0, context=0),
        # the true float32 path that outputs are checked against
        dict(name="block_float32", kind="block", dtype="float32", width=2048, heads=16, kv_heads=4,
             dim=128, ff=6144, requests=2, tokens=301, spread=0.3, context=0),
        # routed experts beside a shared feed-forward: a prompt, and a decoding batch
        dict(name="experts_prompt", kind="experts", width=2048, experts=32, top=4, ff=768, shared=3072,
             scores="chosen", groups=1, keep=1, gated=True, requests=1, tokens=2048),
        dict(name="experts_batch", kind="experts", width=2048, experts=32, top=4, ff=768, shared=3072,
             scores="sigmoid", groups=4, keep=2, gated=True, requests=64, tokens=1),
        # windowed attention with a sink: prompts of unlike lengths, some of them continued
        dict(name="window_prompt", kind="attention", width=2048, heads=16, kv_heads=4, dim=128, window=1024,
             keep_first=0, sink=True, softcap=0.0, requests=2, tokens=2048, spread=0.5, context=300),
        # causal attention with bounded scores: single tokens of a batch over long contexts
        dict(name="capped_batch", kind="attention", width=4096, heads=16, kv_heads=4, dim=128, window=0,
             keep_first=0, sink=False, softcap=30.0, requests=64, tokens=1, spread=0.5, context=4001),
        # attention over one compressed row a token
        dict(name="latent_prompt", kind="latent", width=2048, heads=16, dim=128, rope=64, rank=512,
             q_rank=1536, requests=1, tokens=2048, spread=0.0, context=0),
        # recurrent layers over prompts, one of them a continued portion
        dict(name="state_space_prompt", kind="state_space", width=2048, heads=64, channels=64, state=128,
             groups=8, requests=1, tokens=2048, spread=0.0, context=0),
        dict(name="delta_prompt", kind="delta", width=2048, heads=16, kv_heads=8, dim=128, channels=128,
             requests=3, tokens=1111, spread=0.7, context=100),
        dict(name="retention_prompt", kind="retention", width=4096, heads=16, dim=128, channels=256,
             requests=1, tokens=4096, spread=0.0, context=0),
    ]


def draw(rng):
    """One more case of the listed ranges: any kind, prompts of 20 to about 3000 tokens in all or
    batches of 8 to 96 single tokens."""
    def log_between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["turn", "block", "block32", "experts", "experts", "attention", "attention",
                       "latent", "state_space", "delta", "retention"])
    wide = rng.random() < 0.4
    width, ff = (4096, 12288) if wide else (2048, 6144)
    batch = rng.random() < 0.3
    if batch:
        step = dict(requests=log_between(8, 96), tokens=1, spread=round(rng.uniform(0, 0.9), 2),
                    context=log_between(64, 4000))
    else:
        requests = rng.choice([1, 1, 2, 3, 5])
        step = dict(requests=requests, tokens=log_between(20, 3000 // requests),
                    spread=round(rng.uniform(0, 0.9), 2), context=rng.choice([0, 0, log_between(5, 1500)]))
    if kind == "turn":
        requests = log_between(1, 32)
        return dict(kind="turn", width=2048, heads=16, kv_heads=4, dim=128, ff=6144, layers=rng.choice([2, 3]),
                    vocab=32768, requests=requests, tokens=log_between(10, 400),
                    spread=round(rng.uniform(0, 0.9), 2), steps=rng.randint(8, 24))
    if kind == "block":
        heads, kv = (32, 8) if wide else (16, 4)
        return dict(kind="block", dtype="bfloat16", width=width, heads=heads, kv_heads=kv, dim=128, ff=ff, **step)
    if kind == "block32":
        return dict(kind="block", dtype="float32", width=2048, heads=16, kv_heads=4, dim=128, ff=6144,
                    requests=rng.choice([1, 2, 3]), tokens=log_between(4, 180), spread=0.4,
                    context=rng.choice([0, log_between(5, 200)]))
    if kind == "experts":
        scores = rng.choice(["chosen", "all", "sigmoid"])
        groups, keep = rng.choice([(1, 1), (4, 2)]) if scores != "chosen" else (1, 1)
        return dict(kind="experts", width=width, experts=rng.choice([16, 32, 32, 64]), top=rng.choice([2, 4, 4, 6]),
                    ff=rng.choice([512, 768, 768, 1024, 1536]), shared=rng.choice([0, ff // 2]), scores=scores,
                    groups=groups, keep=keep, gated=rng.random() < 0.75, requests=step["requests"],
                    tokens=step["tokens"])
    if kind == "attention":
        window = rng.choice([0, 0, 512, 1024])
        return dict(kind="attention", width=width, heads=16, kv_heads=rng.choice([2, 4, 4, 8]),
                    dim=rng.choice([64, 128, 128]), window=window, keep_first=4 if window and rng.random() < 0.4 else 0,
                    sink=rng.random() < 0.5, softcap=rng.choice([0.0, 0.0, 30.0]), **step)
    if kind == "latent":
        return dict(kind="latent", width=width, heads=16, dim=128, rope=64, rank=512,
                    q_rank=rng.choice([0, 3 * width // 4]), **step)
    if kind == "state_space":
        return dict(kind="state_space", width=2048, heads=rng.choice([32, 64]), channels=64, state=128, groups=8,
                    **step)
    if kind == "delta":
        return dict(kind="delta", width=width, heads=16, kv_heads=rng.choice([8, 16]), dim=128, channels=128, **step)
    return dict(kind="retention", width=width, heads=width // 256, dim=128, channels=256, **step)


# ------------------------------------------------------------------------------ the step


def _lengths(case):
    """(tokens each request brings, tokens each has in the cache already)."""
    n, r, s = case["tokens"], case["requests"], case.get("spread", 0.0)
    shares = [1.0 - s * i / r for i in range(r)]
    return ([max(1, round(n * f)) for f in shares],
            [round(case.get("context", 0) * f) for f in shares])


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else BF


def _generator(seed, salt):
    return torch.Generator(device=DEV).manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFF)


def _step(case):
    extents, firsts = _lengths(case)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)            # noqa: E731
    starts = [0]
    for n in extents:
        starts.append(starts[-1] + n)
    positions = torch.cat([torch.arange(f, f + n, dtype=torch.int32, device=DEV)
                           for n, f in zip(extents, firsts)])
    requests = len(extents)
    seq = torch.repeat_interleave(torch.arange(requests, dtype=torch.int32, device=DEV), t(extents).long())
    return StepContext(
        num_tokens=starts[-1], num_seqs=requests, token_ids=torch.zeros_like(positions), positions=positions,
        seq_ids=seq, q_start=t(starts), context_lens=t([f + n for n, f in zip(extents, firsts)]),
        state_slots=t([i + 1 for i in range(requests)]), logit_rows=t([]), act_dtype=_dtype(case), extents=extents,
        first_positions=firsts, max_extent=max(extents), max_context=max(f + n for n, f in zip(extents, firsts)),
        decode_only=max(extents) == 1)


def _pages(case, seed):
    """Block tables (pages in no order, page 0 the one nobody owns) and a slot per token."""
    extents, firsts = _lengths(case)
    counts = [-(-(f + n) // PAGE) for n, f in zip(extents, firsts)]
    order = torch.randperm(sum(counts), generator=_generator(seed, 1), device=DEV).to(torch.int32) + 1
    table = torch.zeros((len(counts), max(counts)), dtype=torch.int32, device=DEV)
    slots, at = [], 0
    for i, (c, n, f) in enumerate(zip(counts, extents, firsts)):
        table[i, :c] = order[at:at + c]
        at += c
        p = torch.arange(f, f + n, device=DEV)
        slots.append(table[i][p // PAGE].long() * PAGE + p % PAGE)
    return table, torch.cat(slots).to(torch.int32), sum(counts) + 1


def _planes(case, seed, shapes, pages):
    """The cache planes of a call: earlier tokens' rows drawn, the unowned page NaN."""
    g, out = _generator(seed, 2), []
    for heads, width in shapes:
        p = torch.randn((pages, heads, PAGE, width), generator=g, device=DEV).to(_dtype(case))
        p[0] = float("nan")
        out.append(p)
    return out


def _rows(case, seed):
    n = sum(_lengths(case)[0])
    return torch.randn((n, case["width"]), generator=_generator(seed, 3), device=DEV)


def _state(case, seed, floats):
    """State rows, a spare one first; drawn for requests that are continued, zero for new ones."""
    s = torch.randn((case["requests"] + 1, floats), generator=_generator(seed, 4), device=DEV)
    return s * 0.3 if case.get("context") else s * 0.0


# --------------------------------------------------------------------------- the weights


def _weights(case, seed):
    """{role: tensor} of the case's part, stored as a checkpoint's tensors are bound."""
    g, d, kind = _generator(seed, 5), case["width"], case["kind"]
    normal = lambda *s: torch.randn(s, generator=g, device=DEV)             # noqa: E731
    uniform = lambda lo, hi, *s: torch.rand(s, generator=g, device=DEV) * (hi - lo) + lo   # noqa: E731
    matrix = lambda n, k: (normal(n, k) * k ** -0.5).to(_dtype(case))       # noqa: E731
    gain = lambda n: 1.0 + 0.1 * normal(n)                                  # noqa: E731

    def step_bias(n):                  # softplus of it spreads over 0.001 .. 0.1
        dt = torch.exp(uniform(math.log(1e-3), math.log(0.1), n))
        return dt + torch.log(-torch.expm1(-dt))
    if kind == "block":
        qw, kw, ff = case["heads"] * case["dim"], case["kv_heads"] * case["dim"], case["ff"]
        return dict(mixer_norm=gain(d), ffn_norm=gain(d), q=matrix(qw, d), k=matrix(kw, d), v=matrix(kw, d),
                    o=matrix(d, qw), q_norm=gain(case["dim"]), k_norm=gain(case["dim"]), gate=matrix(ff, d),
                    up=matrix(ff, d), down=matrix(d, ff))
    if kind == "experts":
        f, E = case["ff"], case["experts"]
        w = {}
        for e in range(E):
            if case["gated"]:
                w[f"expert_gate.{e}"] = matrix(f, d)
            w[f"expert_up.{e}"], w[f"expert_down.{e}"] = matrix(f, d), matrix(d, f)
        w["router"] = normal(E, d) * d ** -0.5
        if case["shared"]:
            w.update(gate=matrix(case["shared"], d), up=matrix(case["shared"], d), down=matrix(d, case["shared"]))
        return w
    if kind == "attention":
        qw, kw = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        w = dict(q=matrix(qw, d), k=matrix(kw, d), v=matrix(kw, d), o=matrix(d, qw), q_bias=0.1 * normal(qw),
                 k_bias=0.1 * normal(kw), v_bias=0.1 * normal(kw))
        if case["sink"]:
            w["sink"] = normal(case["heads"])
        return w
    if kind == "latent":
        H, dn, dr, rank, qr = case["heads"], case["dim"], case["rope"], case["rank"], case["q_rank"]
        w = dict(kv_down=matrix(rank + dr, d), kv_norm=gain(rank), k_up=matrix(H * dn, rank),
                 v_up=matrix(H * dn, rank), o=matrix(d, H * dn))
        if qr:
            w.update(q_down=matrix(qr, d), q_down_norm=gain(qr), q_up=matrix(H * (dn + dr), qr))
        else:
            w["q"] = matrix(H * (dn + dr), d)
        return w
    if kind == "state_space":
        H, P, N, G = case["heads"], case["channels"], case["state"], case["groups"]
        inner, C = H * P, H * P + 2 * G * N
        return {"in": matrix(2 * inner + 2 * G * N + H, d), "conv": 0.5 * normal(C, 4), "conv_bias": 0.1 * normal(C),
                "dt_bias": step_bias(H), "a_log": torch.log(uniform(1.0, 16.0, H)), "d": gain(H),
                "norm": gain(inner), "o": matrix(d, inner)}
    if kind == "delta":
        H, kw, vw = case["heads"], case["kv_heads"] * case["dim"], case["heads"] * case["channels"]
        return dict(q=matrix(kw, d), k=matrix(kw, d), v=matrix(vw, d), q_conv=0.5 * normal(kw, 4),
                    k_conv=0.5 * normal(kw, 4), v_conv=0.5 * normal(vw, 4), a=matrix(H, d), b=matrix(H, d),
                    gate=matrix(vw, d), a_log=torch.log(uniform(1.0, 16.0, H)), dt_bias=step_bias(H),
                    norm=gain(case["channels"]), o=matrix(d, vw))
    qk, vw = case["heads"] * case["dim"], case["heads"] * case["channels"]
    return dict(q=matrix(qk, d), k=matrix(qk, d), v=matrix(vw, d), gate=matrix(vw, d), o=matrix(d, vw))


def _next_norm(case, seed):
    return {"next_norm": 1.0 + 0.1 * torch.randn(case["width"], generator=_generator(seed, 6), device=DEV)}


def _decay(case):
    n = case["heads"]
    return tuple(1.0 - 2.0 ** (-5 - 5 * i / max(1, n - 1)) for i in range(n))


def _part(case):
    """The case's part, made from its spec."""
    kind, d = case["kind"], case["width"]
    names = lambda *roles: tuple((r, r) for r in roles)                     # noqa: E731
    if kind == "block":
        mixer = MixerSpec("gqa_attention", num_heads=case["heads"], num_kv_heads=case["kv_heads"],
                          head_dim=case["dim"], qk_norm=True, norm_eps=EPS,
                          position=PositionSpec("rope_half_split", rotary_dim=case["dim"], theta=THETA),
                          tensors=names("q", "k", "v", "o", "q_norm", "k_norm"))
        ffn = FeedForwardSpec("swiglu", intermediate_size=case["ff"], tensors=names("gate", "up", "down"))
        spec = LayerSpec("prenorm_residual", "", mixer, ffn, NormSpec("rmsnorm", EPS), names("mixer_norm", "ffn_norm"))
        return BLOCKS.get(spec.block)(spec, d, DEV)
    if kind == "experts":
        shared = FeedForwardSpec("swiglu", intermediate_size=case["shared"], tensors=names("gate", "up", "down")) \
            if case["shared"] else None
        roles = [("expert_up", "expert_up.{e}"), ("expert_down", "expert_down.{e}"), ("router", "router")]
        if case["gated"]:
            roles.append(("expert_gate", "expert_gate.{e}"))
        spec = FeedForwardSpec("routed_experts", intermediate_size=case["ff"], experts=case["experts"],
                               top=case["top"], shared=shared, gated=case["gated"], router_scores=case["scores"],
                               router_groups=(case["groups"], case["keep"]) if case["groups"] > 1 else None,
                               tensors=tuple(roles))
        return FEED_FORWARDS.get(spec.kind)(spec, d, "", DEV)
    if kind == "attention":
        spec = MixerSpec("sink_attention", num_heads=case["heads"], num_kv_heads=case["kv_heads"],
                         head_dim=case["dim"], window=case["window"] or None, keep_first=case["keep_first"],
                         bias=True, sink=case["sink"], softcap=case["softcap"] or None,
                         position=PositionSpec("rope_half_split", rotary_dim=case["dim"] // 2, theta=THETA),
                         tensors=names("q", "k", "v", "o", "q_bias", "k_bias", "v_bias", "sink"))
    elif kind == "latent":
        spec = MixerSpec("latent_attention", num_heads=case["heads"], head_dim=case["dim"], value_dim=case["dim"],
                         rope_dim=case["rope"], latent_rank=case["rank"], query_rank=case["q_rank"], norm_eps=EPS,
                         position=PositionSpec("rope_half_split", rotary_dim=case["rope"], theta=THETA),
                         tensors=names("q", "q_down", "q_down_norm", "q_up", "kv_down", "kv_norm", "k_up", "v_up", "o"))
    elif kind == "state_space":
        spec = MixerSpec("selective_state_space", num_heads=case["heads"], value_dim=case["channels"],
                         head_dim=case["state"], num_kv_heads=case["groups"], conv_taps=4,
                         norm_groups=case["groups"], norm_eps=EPS,
                         tensors=names("in", "conv", "conv_bias", "dt_bias", "a_log", "d", "norm", "o"))
    elif kind == "delta":
        spec = MixerSpec("gated_delta", num_heads=case["heads"], num_kv_heads=case["kv_heads"],
                         head_dim=case["dim"], value_dim=case["channels"], conv_taps=4, norm_eps=EPS,
                         tensors=names("q", "k", "v", "q_conv", "k_conv", "v_conv", "a", "b", "gate", "a_log",
                                       "dt_bias", "norm", "o"))
    else:
        spec = MixerSpec("retention", num_heads=case["heads"], head_dim=case["dim"], value_dim=case["channels"],
                         decay=_decay(case), output_gate=True, norm_eps=EPS,
                         position=PositionSpec("rope_half_split", rotary_dim=case["dim"], theta=THETA),
                         tensors=names("q", "k", "v", "gate", "o"))
    return MIXERS.get(spec.kind)(spec, d, "", DEV)


# --------------------------------------------------------------------------- whole calls


def _turn_weights(case, seed):
    g, d, V = _generator(seed, 5), case["width"], case["vocab"]
    qw, kw, ff = case["heads"] * case["dim"], case["kv_heads"] * case["dim"], case["ff"]
    matrix = lambda n, k: (torch.randn((n, k), generator=g, device=DEV) * k ** -0.5).to(BF)   # noqa: E731
    gain = lambda n: 1.0 + 0.1 * torch.randn((n,), generator=g, device=DEV)                  # noqa: E731
    w = {"model.embed_tokens.weight": matrix(V, d) * 16}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        w.update({p + "input_layernorm.weight": gain(d), p + "post_attention_layernorm.weight": gain(d),
                  p + "self_attn.q_proj.weight": matrix(qw, d), p + "self_attn.k_proj.weight": matrix(kw, d),
                  p + "self_attn.v_proj.weight": matrix(kw, d), p + "self_attn.o_proj.weight": matrix(d, qw),
                  p + "self_attn.q_norm.weight": gain(case["dim"]), p + "self_attn.k_norm.weight": gain(case["dim"]),
                  p + "mlp.gate_proj.weight": matrix(ff, d), p + "mlp.up_proj.weight": matrix(ff, d),
                  p + "mlp.down_proj.weight": matrix(d, ff)})
    w["model.norm.weight"] = gain(d)
    w["lm_head.weight"] = matrix(V, d)
    return w


def _turn_tokens(case, seed):
    """Per request: the prompt and the tokens decoded after it."""
    extents, _ = _lengths(case)
    g = torch.Generator().manual_seed(int(seed) * 7919 + 17)
    ids = [torch.randint(0, case["vocab"], (n + case["steps"],), generator=g).tolist() for n in extents]
    return [t[:n] for t, n in zip(ids, extents)], [t[n:] for t, n in zip(ids, extents)]


def _turn_prepare(case, seed):
    from tgo_b200.api import LoadedModel
    from tgo_b200.engine.model import Model
    from tgo_b200.registry import model_spec_from_config
    config = dict(architectures=["Qwen3ForCausalLM"], hidden_size=case["width"], num_hidden_layers=case["layers"],
                  num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=case["dim"],
                  intermediate_size=case["ff"], vocab_size=case["vocab"], rms_norm_eps=EPS, rope_theta=THETA,
                  tie_word_embeddings=False, max_position_embeddings=8192)
    model = Model(model_spec_from_config(config), BF, DEV)
    model.bind(_turn_weights(case, seed))
    prompts, rest = _turn_tokens(case, seed)
    tokens = sum(-(-(len(p) + case["steps"]) // PAGE) * PAGE for p in prompts)
    engine = LoadedModel(model, config, "").new_engine(page_size=PAGE, max_tokens=tokens, num_slots=len(prompts))
    return dict(engine=engine, prompts=prompts, rest=rest, steps=case["steps"])


def _turn_run(s):
    engine, prompts, rest = s["engine"], s["prompts"], s["rest"]
    for i in range(len(prompts)):
        engine.admit(i)
    out = [engine.step([StepEntry(i, p, [len(p) - 1]) for i, p in enumerate(prompts)]).clone()]
    for j in range(s["steps"]):
        out.append(engine.step([StepEntry(i, [r[j]], [0]) for i, r in enumerate(rest)]).clone())
    for i in range(len(prompts)):
        engine.finish(i)
    return {"prompt": out[0], "decoded": out[1:]}


# --------------------------------------------------------------------- prepare, run, work


def prepare(case, seed):
    kind = case["kind"]
    if kind == "turn":
        return _turn_prepare(case, seed)
    part, ctx = _part(case), _step(case)
    part.bind(_weights(case, seed))
    x = _rows(case, seed)
    s = dict(kind=kind, part=part, ctx=ctx, cache=LayerCache(page_size=PAGE))
    cache = s["cache"]
    if kind == "block":
        s["stream"], s["h"] = x, torch.empty_like(x)
        s["norm"] = NORMS.get("rmsnorm")(NormSpec("rmsnorm", EPS), case["width"], "next_norm")
        s["norm"].bind(_next_norm(case, seed))
    else:
        s["x"] = x.to(_dtype(case))
    shapes = {"block": [(case.get("kv_heads"), case.get("dim"))] * 2,
              "attention": [(case.get("kv_heads"), case.get("dim"))] * 2,
              "latent": [(1, case.get("rank", 0) + case.get("rope", 0))]}.get(kind)
    if shapes:
        cache.block_tables, cache.slots, pages = _pages(case, seed)
        planes = _planes(case, seed, shapes, pages)
        if kind == "latent":
            planes[0][:, :, :, case["rank"]:] *= 0.5
        cache.planes = torch.stack(planes)
        cache.group = 0
    if kind in ("state_space", "delta", "retention"):
        need = part.state_need().shape
        floats = 1
        for n in need:
            floats *= n
        cache.state = _state(case, seed, floats).view(case["requests"] + 1, *need)
    return s


def run(s):
    """One pass of the call. The step's context is used as a model uses it: every layer of a step
    shares it; a block's stream starts from the same rows each time."""
    kind = s.get("kind")
    if kind is None:
        return _turn_run(s)
    part, ctx, cache = s["part"], s["ctx"], s["cache"]
    if kind == "block":
        # the next layer's norm adds what the block leaves pending
        h, pending = part.forward(s["h"].copy_(s["stream"]), None, ctx, cache)
        rows = s["norm"].forward(h, pending, ctx.act_dtype)
        return {"stream": h, "rows": rows, "cache": cache.planes}
    if kind == "experts":
        return {"out": part.forward(s["x"], ctx)}
    out = {"out": part.forward(s["x"], ctx, cache)}
    if cache.planes is not None:
        out["cache"] = cache.planes
    if cache.state is not None:
        out["state"] = cache.state
    return out


def _keys_read(case):
    """(query-key pairs, keys of the cache read) of an attention step."""
    pairs = read = 0
    window, keep = case.get("window", 0), case.get("keep_first", 0)
    for n, f in zip(*_lengths(case)):
        for p in range(f, f + n):
            pairs += p + 1 if not window else min(p + 1, window) + min(keep, max(0, p + 1 - window))
        read += f + n if not window else min(f + n, window + n + keep)
    return pairs, read


def work(case):
    kind, d = case["kind"], case["width"]
    extents, _ = _lengths(case)
    T, e = sum(extents), 4 if case.get("dtype") == "float32" else 2
    io = 2 * T * d * e
    if kind == "turn":
        H, G, dim, ff, V = (case[k] for k in ("heads", "kv_heads", "dim", "ff", "vocab"))
        layer = 2 * H * dim * d + 2 * G * dim * d + 3 * ff * d
        pairs = sum(sum(range(1, n + 1)) + case["steps"] * (n + case["steps"] / 2) for n in extents)
        tokens, B = T + case["steps"] * len(extents), len(extents)
        weights = 2 * (layer * case["layers"] + V * d) * (1 + case["steps"])
        cache = case["layers"] * 4 * G * dim * sum(case["steps"] * (n + case["steps"] / 2) for n in extents)
        logits = 4 * V * B * (1 + case["steps"])
        return {"bytes": weights + cache + logits,
                "flops": 2 * tokens * layer * case["layers"] + 4 * H * dim * pairs * case["layers"] +
                2 * B * (1 + case["steps"]) * V * d}
    if kind == "experts":
        f, shared, n = case["ff"], case["shared"], 3 if case["gated"] else 2
        used = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** T)
        weights = 2 * (used * n * f * d + 3 * shared * d) + 4 * case["experts"] * d
        return {"bytes": io + weights,
                "flops": 2 * T * d * (case["experts"] + case["top"] * n * f + 3 * shared)}
    if kind in ("block", "attention"):
        qw, kw = case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        ff = 3 * case["ff"] if kind == "block" else 0
        pairs, read = _keys_read(case)
        n = d * (2 * qw + 2 * kw + ff)
        return {"bytes": (2 * T * d * 4 if kind == "block" else io) + e * n + 2 * e * kw * (read + T),
                "flops": 2 * T * n + 4 * qw * pairs}
    if kind == "latent":
        H, dn, dr, rank, qr = (case[k] for k in ("heads", "dim", "rope", "rank", "q_rank"))
        pairs, read = _keys_read(case)
        n = d * (rank + dr + H * dn) + 2 * H * dn * rank + (qr * (d + H * (dn + dr)) if qr else d * H * (dn + dr))
        return {"bytes": io + 2 * n + 2 * (rank + dr) * (read + T), "flops": 2 * T * n + 2 * H * (2 * rank + dr) * pairs}
    if kind == "state_space":
        H, P, N, G = (case[k] for k in ("heads", "channels", "state", "groups"))
        n, floats = d * (3 * H * P + 2 * G * N + H), H * N * P + 3 * (H * P + 2 * G * N)
        return {"bytes": io + 2 * n + 8 * floats * case["requests"], "flops": 2 * T * n + 6 * T * H * N * P}
    if kind == "delta":
        H, kw, dk, dv = case["heads"], case["kv_heads"] * case["dim"], case["dim"], case["channels"]
        n, floats = d * (2 * kw + 3 * H * dv + 2 * H), H * dk * dv + 3 * (2 * kw + H * dv)
        return {"bytes": io + 2 * n + 8 * floats * case["requests"], "flops": 2 * T * n + 6 * T * H * dk * dv}
    H, dk, dv = case["heads"], case["dim"], case["channels"]
    n = d * (2 * H * dk + 3 * H * dv)
    return {"bytes": io + 2 * n + 8 * H * dk * dv * case["requests"], "flops": 2 * T * n + 4 * T * H * dk * dv}


def tolerance(case):
    """About four times what the start shows against 64 bits (or, where the state's float32 sums are
    compared, their order): bfloat16 rows rounded between kernels; sums in 32 bits."""
    if case.get("dtype") == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "turn":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.015, "max": 0.2}


# -------------------------------------------------------------------------- in 64 bits


def _norm(x, gain, eps=EPS):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _turned(x, positions, rot):
    """The first `rot` channels of x [T, heads, dim] turned, channel i with i + rot/2."""
    f = THETA ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64, device=DEV) / rot)
    a = positions.double()[:, None] * f[None]
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    lo, hi = x[..., :rot // 2], x[..., rot // 2:rot]
    return torch.cat([lo * c - hi * s, hi * c + lo * s, x[..., rot:]], -1)


def _attend(q, keys, values, first, scale, window=0, keep=0, sink=None, cap=0.0):
    """q [n, H, dk] at positions first.. over keys [m, G, dk], values [m, G, dv]; [n, H, dv]."""
    n, H, _ = q.shape
    m, G, _ = keys.shape
    out = torch.empty((n, H, values.shape[-1]), dtype=torch.float64, device=DEV)
    for lo in range(0, n, 512):
        hi = min(n, lo + 512)
        i = torch.arange(first + lo, first + hi, device=DEV)[:, None]
        j = torch.arange(m, device=DEV)[None]
        seen = j <= i
        if window:
            seen &= (i - j < window) | (j < keep)
        for g in range(G):
            heads = slice(g * (H // G), (g + 1) * (H // G))
            s = torch.einsum("nhd,md->hnm", q[lo:hi, heads], keys[:, g]) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(~seen, float("-inf"))
            if sink is not None:
                s = torch.cat([s, sink[heads].view(-1, 1, 1).expand(-1, hi - lo, 1)], -1)
            w = torch.softmax(s, -1)[..., :m]
            out[lo:hi, heads] = torch.einsum("hnm,md->nhd", w, values[:, g])
    return out


def _cached(plane, table, count):
    """The first `count` rows [count, heads, width] of a request's pages."""
    rows = plane[table.long()].transpose(1, 2).reshape(-1, plane.shape[1], plane.shape[3])
    return rows[:count].double()


def _attention64(case, x, w, seed, norms=None):
    """Rows [T, H dim] of a grouped-query attention before its output product."""
    H, G, dim = case["heads"], case["kv_heads"], case["dim"]
    extents, firsts = _lengths(case)
    q, k, v = (x @ w[r].T + (w[r + "_bias"] if r + "_bias" in w else 0.0) for r in ("q", "k", "v"))
    q, k, v = q.view(-1, H, dim), k.view(-1, G, dim), v.view(-1, G, dim)
    rot = dim // 2
    if norms:
        q, k, rot = _norm(q, w["q_norm"]), _norm(k, w["k_norm"]), dim
    out, at = torch.empty_like(q), 0
    if any(firsts):
        table, _, pages = _pages(case, seed)
        planes = _planes(case, seed, [(G, dim)] * 2, pages)
    for i, (n, f) in enumerate(zip(extents, firsts)):
        p = torch.arange(f, f + n, device=DEV)
        sl = slice(at, at + n)
        keys, values = _turned(k[sl], p, rot), v[sl]
        if f:
            keys = torch.cat([_cached(planes[0], table[i], f), keys])
            values = torch.cat([_cached(planes[1], table[i], f), values])
        out[sl] = _attend(_turned(q[sl], p, rot), keys, values, f, dim ** -0.5, case.get("window", 0),
                          case.get("keep_first", 0), w.get("sink"), case.get("softcap", 0.0))
        at += n
    return out.reshape(-1, H * dim)


def _dense64(x, w):
    return (_silu(x @ w["gate"].T) * (x @ w["up"].T)) @ w["down"].T


def _experts64(case, x, w):
    E, top = case["experts"], case["top"]
    z = x @ w["router"].T
    if case["scores"] == "chosen":
        ids = torch.topk(z, top, -1).indices
        weight = torch.softmax(torch.gather(z, 1, ids), -1)
    else:
        s = torch.softmax(z, -1) if case["scores"] == "all" else torch.sigmoid(z)
        choice = s.clone()
        if case["groups"] > 1:
            runs = s.view(-1, case["groups"], E // case["groups"])
            strength = torch.topk(runs, min(2, runs.shape[-1]), -1).values.sum(-1)
            kept = torch.topk(strength, case["keep"], -1).indices
            mask = torch.zeros_like(strength, dtype=torch.bool).scatter_(1, kept, True)
            choice = runs.masked_fill(~mask[..., None], float("-inf")).reshape(-1, E)
        ids = torch.topk(choice, top, -1).indices
        weight = torch.gather(s, 1, ids)
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    out = torch.zeros_like(x)
    for e in range(E):
        row, place = torch.nonzero(ids == e, as_tuple=True)
        if row.numel():
            up = x[row] @ w[f"expert_up.{e}"].double().T
            h = _silu(x[row] @ w[f"expert_gate.{e}"].double().T) * up if case["gated"] else _silu(up)
            out.index_add_(0, row, (h @ w[f"expert_down.{e}"].double().T) * weight[row, place][:, None])
    if case["shared"]:
        out += _dense64(x, {r: w[r].double() for r in ("gate", "up", "down")})
    return out


def _latent64(case, x, w, seed):
    H, dn, dr, rank = case["heads"], case["dim"], case["rope"], case["rank"]
    extents, firsts = _lengths(case)
    q = _norm(x @ w["q_down"].T, w["q_down_norm"]) @ w["q_up"].T if case["q_rank"] else x @ w["q"].T
    q = q.view(-1, H, dn + dr)
    y = x @ w["kv_down"].T
    c, r = _norm(y[:, :rank], w["kv_norm"]), y[:, rank:]
    k_up, v_up = w["k_up"].view(H, dn, rank), w["v_up"].view(H, dn, rank)
    out, at = [], 0
    if any(firsts):
        table, _, pages = _pages(case, seed)
        plane = _planes(case, seed, [(1, rank + dr)], pages)[0]
        plane[:, :, :, rank:] *= 0.5
    for i, (n, f) in enumerate(zip(extents, firsts)):
        p = torch.arange(f, f + n, device=DEV)
        sl = slice(at, at + n)
        rows = torch.cat([c[sl], _turned(r[sl][:, None], p, dr)[:, 0]], -1)
        if f:
            rows = torch.cat([_cached(plane, table[i], f)[:, 0], rows])
        qa = torch.cat([torch.einsum("nhd,hdr->nhr", q[sl][..., :dn], k_up), _turned(q[sl][..., dn:], p, dr)], -1)
        a = _attend(qa, rows[:, None], rows[:, None, :rank], f, (dn + dr) ** -0.5)
        out.append(torch.einsum("nhr,hdr->nhd", a, v_up).reshape(n, H * dn))
        at += n
    return torch.cat(out) @ w["o"].T


def _convolved(rows, kept, taps):
    """silu of the causal convolution of rows [n, C] after the kept [3, C]; and what is kept next."""
    full = torch.cat([kept, rows])
    n, k = rows.shape[0], taps.shape[1]
    return sum(full[j:j + n] * taps[:, j] for j in range(k)), full[-(k - 1):]


def _recurrent64(case, x, w, seed):
    """(rows before the output product, state rows) of a recurrent mixer."""
    kind, H, dv = case["kind"], case["heads"], case["channels"]
    extents, firsts = _lengths(case)
    dk = case["state"] if kind == "state_space" else case["dim"]
    mem = H * dk * dv
    if kind == "state_space":
        inner, gn = H * dv, case["groups"] * dk
        C = inner + 2 * gn
        z = x @ w["in"].T
    elif kind == "delta":
        kw, inner = case["kv_heads"] * dk, H * dv
        C = 2 * kw + inner
        raw = torch.cat([x @ w[r].T for r in ("q", "k", "v")], -1)
        taps = torch.cat([w[r] for r in ("q_conv", "k_conv", "v_conv")])
        beta = torch.sigmoid(x @ w["b"].T)
        g = torch.exp(-torch.exp(w["a_log"]) * torch.nn.functional.softplus(x @ w["a"].T + w["dt_bias"]))
        z = x @ w["gate"].T
    else:
        C, inner = 0, H * dv
        decay = torch.tensor(_decay(case), dtype=torch.float64, device=DEV)[:, None, None]
    floats = mem + 3 * C
    state = _state(case, seed, floats).double()
    out, at = torch.empty((x.shape[0], H, dv), dtype=torch.float64, device=DEV), 0
    for i, (n, f) in enumerate(zip(extents, firsts)):
        sl, S = slice(at, at + n), state[i + 1, :mem].view(H, dk, dv).clone()
        kept = state[i + 1, mem:].view(3, C) if C else None
        if kind == "state_space":
            conv, kept = _convolved(z[sl, inner:inner + C], kept, w["conv"])
            conv = _silu(conv + w["conv_bias"])
            u = conv[:, :inner].view(n, H, dv)
            B, K = (conv[:, inner + j * gn:inner + (j + 1) * gn].view(n, case["groups"], dk)
                    .repeat_interleave(H // case["groups"], 1) for j in (0, 1))
            dt = torch.nn.functional.softplus(z[sl, inner + C:] + w["dt_bias"])
            a = torch.exp(-torch.exp(w["a_log"]) * dt)
            ub = u * dt[..., None]
            for t in range(n):
                S = a[t, :, None, None] * S + B[t][:, :, None] * ub[t][:, None]
                out[at + t] = torch.einsum("hkv,hk->hv", S, K[t]) + w["d"][:, None] * u[t]
        elif kind == "delta":
            conv, kept = _convolved(raw[sl], kept, taps)
            conv = _silu(conv)
            unit = lambda v: v * torch.rsqrt((v * v).sum(-1, keepdim=True) + 1e-6)   # noqa: E731
            G = case["kv_heads"]
            q, k = (unit(conv[:, j * kw:(j + 1) * kw].view(n, G, dk)).repeat_interleave(H // G, 1) for j in (0, 1))
            q, v = q * dk ** -0.5, conv[:, 2 * kw:].view(n, H, dv)
            for t in range(n):
                S = g[at + t][:, None, None] * S
                u = beta[at + t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
                S = S + k[t][:, :, None] * u[:, None]
                out[at + t] = torch.einsum("hkv,hk->hv", S, q[t])
        else:
            p = torch.arange(f, f + n, device=DEV)
            q = _turned((x[sl] @ w["q"].T).view(n, H, dk), p, dk)
            k = _turned((x[sl] @ w["k"].T).view(n, H, dk), p, dk) * dk ** -0.5
            v = (x[sl] @ w["v"].T).view(n, H, dv)
            for t in range(n):
                S = decay * S + k[t][:, :, None] * v[t][:, None]
                out[at + t] = torch.einsum("hkv,hk->hv", S, q[t])
        state[i + 1, :mem] = S.reshape(-1)
        if C:
            state[i + 1, mem:] = kept.reshape(-1)
        at += n
    y = out.reshape(-1, H * dv)
    if kind == "state_space":
        y = y * _silu(z[:, :inner])
        y = _norm(y.view(-1, case["groups"], inner // case["groups"]), 1.0).reshape(-1, inner) * w["norm"]
    elif kind == "delta":
        y = _norm(out, w["norm"]).reshape(-1, inner) * _silu(z)
    else:
        y = _norm(out, 1.0).reshape(-1, inner) * _silu(x @ w["gate"].T)
    return y, state


def _turn64(case, seed):
    w, d = {k: v.double() for k, v in _turn_weights(case, seed).items()}, case["width"]
    prompts, rest = _turn_tokens(case, seed)
    logits = []
    for p, r in zip(prompts, rest):
        h = w["model.embed_tokens.weight"][torch.tensor(p + r, device=DEV)]
        one = dict(case, kind="block", requests=1, tokens=len(p + r), spread=0.0, context=0)
        for i in range(case["layers"]):
            a, m = f"model.layers.{i}.self_attn.", f"model.layers.{i}.mlp."
            lw = {r: w[a + r + "_proj.weight"] for r in ("q", "k", "v", "o")}
            lw.update(q_norm=w[a + "q_norm.weight"], k_norm=w[a + "k_norm.weight"])
            n = _norm(h, w[f"model.layers.{i}.input_layernorm.weight"])
            h = h + _attention64(one, n, lw, seed, norms=True) @ lw["o"].T
            n = _norm(h, w[f"model.layers.{i}.post_attention_layernorm.weight"])
            h = h + _dense64(n, {r: w[m + r + "_proj.weight"] for r in ("gate", "up", "down")})
        logits.append(_norm(h[len(p) - 1:], w["model.norm.weight"]) @ w["lm_head.weight"].T)
    at = [torch.stack([l[j] for l in logits]) for j in range(case["steps"] + 1)]
    return {"prompt": at[0], "decoded": at[1:]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "turn":
        return _turn64(case, seed)
    w = _weights(case, seed)
    x = _rows(case, seed)
    if kind == "experts":
        return {"out": _experts64(case, x.to(_dtype(case)).double(), dict(w, router=w["router"].double()))}
    w = {k: v.double() for k, v in w.items()}
    if kind == "block":
        h = x.double()
        h = h + _attention64(case, _norm(h, w["mixer_norm"]), w, seed, norms=True) @ w["o"].T
        h = h + _dense64(_norm(h, w["ffn_norm"]), w)
        return {"stream": h, "rows": _norm(h, _next_norm(case, seed)["next_norm"].double()), "cache": None}
    x = x.to(BF).double()
    if kind == "attention":
        return {"out": _attention64(case, x, w, seed) @ w["o"].T, "cache": None}
    if kind == "latent":
        return {"out": _latent64(case, x, w, seed), "cache": None}
    y, state = _recurrent64(case, x, w, seed)
    return {"out": y @ w["o"].T, "state": state}
