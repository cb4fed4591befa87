"""What a program built on this package has it do, as a list of cases that can be timed and checked.

Most cases are one layer of one of the registered designs, called the way ``parts.registry`` describes: the part is made
from the specification that the design's configuration gives, loads its tensors by name, and runs on a step's batch
against the cache that ``CacheManager`` keeps.  One case is a whole decode step through ``ModelRunner`` and
``DecodeGraph``, which returns the logits.  Layer sizes are those that ``bench.py`` uses ("4b": Qwen3-4B; "2k" and "4k":
the other designs at widths of 2,048 and 4,096).

Steps that the engine replays from captured graphs are captured here too: decode steps, and prompt steps of up to 1,024
tokens (the engine's own limit) for layers whose launches depend on the token count alone.  Longer prompt steps, and
attention over prompts, whose grids follow how the tokens are spread over requests, are launched call by call.

Everything is bfloat16 with float32 accumulation and float32 recurrent state, which is what serving runs; the 32-bit
mode exists to check results against and is not timed.

A case: ``kind`` (which layer), ``size``, ``mode`` ("prompt": portions of several tokens; "decode": one token a
request), ``requests``, ``tokens`` (of a prompt step, all requests together) and ``context`` (tokens that every request
has in the cache before the step, of layers that cache keys).
"""
from __future__ import annotations

import math

import torch

PAGE = 16
EPS = 1e-6
CAPTURED_TOKENS = 1024
DEVICE = "cuda:0"

QWEN3 = {"4b": dict(hidden=2560, heads=32, kv=8, dim=128, ff=9728, vocab=151936, layers=4, theta=1e6, positions=40960)}
SIZES = {
    "2k": dict(width=2048, heads=16, kv=4, ff=8192, experts=32, top=4, expert_ff=2048, ss_heads=64, ss_dim=64, state=128, groups=8,
               lat_heads=16, lat_dim=128, rot=64, vdim=128, kv_rank=512, q_rank=1536, d_heads=16, d_kv=8, rank=16),
    "4k": dict(width=4096, heads=32, kv=8, ff=12288, experts=64, top=6, expert_ff=2048, ss_heads=128, ss_dim=64, state=128, groups=8,
               lat_heads=32, lat_dim=128, rot=64, vdim=128, kv_rank=512, q_rank=1536, d_heads=32, d_kv=16, rank=32),
}


def listed():
    return [
        # the serving loop's own unit: one token for each of eight requests behind 2,048 tokens, logits out
        {"name": "decode step, 8 requests", "kind": "step", "size": "4b", "mode": "decode", "requests": 8, "tokens": 8, "context": 2048},
        # three prompts' portions of unequal length in one step, each behind what earlier portions left in the cache
        {"name": "attention, prompt portions", "kind": "attention", "size": "4b", "mode": "prompt", "requests": 3, "tokens": 2500, "context": 300},
        # a decode batch beyond the streaming kernels' rows, or a short prompt beside running requests
        {"name": "dense feed-forward, 77 rows", "kind": "mlp", "size": "4b", "mode": "prompt", "requests": 1, "tokens": 77, "context": 0},
        # routed experts of a decode step: the weights of the experts hit are what is read
        {"name": "experts, 8 rows", "kind": "experts_shared", "size": "2k", "mode": "decode", "requests": 8, "tokens": 8, "context": 0},
        # routed experts of a prompt step: the largest products of a layer
        {"name": "experts, 2048 rows", "kind": "experts", "size": "4k", "mode": "prompt", "requests": 1, "tokens": 2048, "context": 0},
        # latent attention while generating: sixteen requests, contexts of a long chat
        {"name": "latent attention, 16 requests", "kind": "latent", "size": "4k", "mode": "decode", "requests": 16, "tokens": 16, "context": 3000},
        # the next portions of two prompts through latent attention
        {"name": "latent attention, prompt", "kind": "latent_low_rank", "size": "2k", "mode": "prompt", "requests": 2, "tokens": 1500, "context": 700},
        # a prompt through the state-space mixer
        {"name": "state space, prompt", "kind": "state_space", "size": "4k", "mode": "prompt", "requests": 1, "tokens": 2048, "context": 0},
        # the smallest call: two requests generating through the state-space mixer
        {"name": "state space, 2 requests", "kind": "state_space", "size": "4k", "mode": "decode", "requests": 2, "tokens": 2, "context": 0},
        # two prompts of unequal, odd length through the gated delta rule
        {"name": "gated delta rule, prompts", "kind": "delta", "size": "2k", "mode": "prompt", "requests": 2, "tokens": 1777, "context": 0},
        # a prompt through linear attention with a decay per channel
        {"name": "gated linear attention, prompt", "kind": "gla", "size": "4k", "mode": "prompt", "requests": 1, "tokens": 2048, "context": 0},
        # a prompt portion through differential attention
        {"name": "differential attention, prompt", "kind": "diff", "size": "2k", "mode": "prompt", "requests": 1, "tokens": 1024, "context": 0},
    ]


def draw(rng):
    def spread(lo, hi):                          # even over the logarithm, odd numbers among them
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["step", "attention", "mlp", "experts_shared", "experts", "latent", "latent_low_rank", "state_space", "state_space",
                       "delta", "gla", "diff"])
    size = "4b" if kind in ("step", "attention", "mlp") else "4k" if kind == "state_space" else rng.choice(["2k", "4k"])
    decode = {"step": True, "attention": False, "diff": False}.get(kind, rng.random() < 0.4)
    if decode:
        requests = spread(1, 32)
        return {"kind": kind, "size": size, "mode": "decode", "requests": requests, "tokens": requests,
                "context": spread(64, 4096) if kind in ("step", "latent", "latent_low_rank") else 0}
    tokens = spread(64, 2048 if kind.startswith("experts") else 4096)
    return {"kind": kind, "size": size, "mode": "prompt", "requests": rng.randint(1, 3), "tokens": tokens,
            "context": spread(16, 2048) if kind in ("attention", "latent", "latent_low_rank") else 0}


# -- sizes of a step -------------------------------------------------------------------------------------------------
def portions(case):
    """Tokens that each request brings: equal to one in a decode step, unequal shares of the step's tokens else."""
    R, T = case["requests"], case["tokens"]
    if case["mode"] == "decode":
        return [1] * R
    parts = [T * (r + 1) * 2 // (R * (R + 1)) for r in range(R)]
    parts[-1] += T - sum(parts)
    return parts


def contexts(case):
    """Tokens that each request has in the cache: up to ``context``, unequal."""
    C = case["context"]
    return [C - (r * 61) % (C // 3 + 1) for r in range(case["requests"])]


# -- the designs' own configurations, one layer each ------------------------------------------------------------------
def qwen3_config(z):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=z["vocab"], hidden_size=z["hidden"],
                intermediate_size=z["ff"], num_hidden_layers=z["layers"], num_attention_heads=z["heads"], num_key_value_heads=z["kv"],
                head_dim=z["dim"], max_position_embeddings=z["positions"], rope_theta=z["theta"], rms_norm_eps=EPS,
                tie_word_embeddings=True, attention_bias=False, use_sliding_window=False, hidden_act="silu")


def config_of(case):
    """(config.json's content, what to take of the layer: "mixer", "mixer.1" (second of two side by side) or "feed_forward")."""
    kind = case["kind"]
    if kind in ("step", "attention", "mlp"):
        return qwen3_config(QWEN3[case["size"]]), "mixer" if kind == "attention" else "feed_forward"
    z = SIZES[case["size"]]
    dense = {"kind": "dense", "ff": z["ff"]}
    top = {"vocab": 512, "width": z["width"], "norm": {"eps": EPS}}
    router = {"experts": z["experts"], "top": z["top"], "groups": {"count": 4, "keep": 2}}
    ssm = {"heads": z["ss_heads"], "vdim": z["ss_dim"], "state": z["state"], "groups": z["groups"], "conv": 4, "norm_groups": z["groups"]}
    lat = {"heads": z["lat_heads"], "dim": z["lat_dim"], "rot_dim": z["rot"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
           "scale": (z["lat_dim"] + z["rot"]) ** -0.5}
    if kind == "state_space":
        layer = {"type": "mamba2", "mixer": ssm, "mlp": dense}
        return dict(top, architecture="Pepolorn", layers=[layer]), "mixer"
    if kind == "experts":
        moe = {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "router": router}
        return dict(top, architecture="Pepolorn", layers=[{"type": "mamba2", "mixer": ssm, "mlp": moe}]), "feed_forward"
    if kind == "latent_low_rank":
        m = dict(lat, q_rank=z["q_rank"], rot=dict(LOW_RANK_ROT, dims=z["rot"]))
        return dict(top, architecture="Kolisun", layers=[{"type": "latent_attention", "mixer": m, "mlp": dense}]), "mixer"
    if kind in ("latent", "gla", "experts_shared"):
        if kind == "gla":
            layer = {"type": "gla", "mixer": {"heads": z["lat_heads"], "dim": 128, "vdim": 128, "tau": 16.0}, "mlp": dense}
        else:
            moe = {"kind": "moe", "expert": {"ff": z["expert_ff"]}, "shared": {"ff": z["expert_ff"]}, "router": dict(router, scale=1.5)}
            layer = {"type": "latent_attention", "mixer": dict(lat, rot={"dims": z["rot"], "base": 100000.0}), "mlp": moe}
        return dict(top, architecture="Nulilix", layers=[layer]), "feed_forward" if kind == "experts_shared" else "mixer"
    if kind == "delta":
        par = {"left": {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                        "mask": {"size": 1024, "keep_first": 64}},
               "right": {"heads": z["d_heads"], "kv_heads": z["d_kv"], "dim": 128, "vdim": 128, "conv": 4}}
        return dict(top, architecture="Nedesun", residual_mult=0.5, embedding={"scale": 1.0},
                    layers=[{"type": "parallel", "mixer": par, "mlp": dense}]), "mixer.1"
    if kind == "diff":
        m = {"heads": z["heads"], "kv_heads": z["kv"], "dim": 64, "vdim": 128, "scale": 64 ** -0.5, "diff": 0.5,
             "q_temp": {"coef": 0.1, "every": 512}}
        return dict(top, architecture="Pabelix", layers=[{"type": "attention", "mixer": m, "mlp": dict(dense, limit=7.0)}]), "mixer"
    raise ValueError(f"unknown kind {kind!r}")


LOW_RANK_ROT = {"base": 10000.0, "scaling": {"factor": 40.0, "original": 4096, "fast": 32.0, "slow": 1.0}}


def tensor_shapes(case):
    """{name: (shape, how it is drawn)} of the layer's tensors, as a checkpoint names them below the layer's prefix."""
    kind = case["kind"]
    if kind in ("step", "attention", "mlp"):
        z = QWEN3[case["size"]]
        D, q, kv = z["hidden"], z["heads"] * z["dim"], z["kv"] * z["dim"]
        att = {"q_proj.weight": ((q, D), "matrix"), "k_proj.weight": ((kv, D), "matrix"), "v_proj.weight": ((kv, D), "matrix"),
               "o_proj.weight": ((D, q), "matrix"), "q_norm.weight": ((z["dim"],), "norm"), "k_norm.weight": ((z["dim"],), "norm")}
        mlp = {"gate_proj.weight": ((z["ff"], D), "matrix"), "up_proj.weight": ((z["ff"], D), "matrix"), "down_proj.weight": ((D, z["ff"]), "matrix")}
        if kind != "step":
            return att if kind == "attention" else mlp
        out = {"model.embed_tokens.weight": ((z["vocab"], D), "table"), "model.norm.weight": ((D,), "norm")}
        for i in range(z["layers"]):
            p = f"model.layers.{i}."
            out.update({p + "self_attn." + n: v for n, v in att.items()})
            out.update({p + "mlp." + n: v for n, v in mlp.items()})
            out.update({p + "input_layernorm.weight": ((D,), "norm"), p + "post_attention_layernorm.weight": ((D,), "norm")})
        return out
    z = SIZES[case["size"]]
    D = z["width"]
    if kind == "state_space":
        inner, ch = z["ss_heads"] * z["ss_dim"], z["ss_heads"] * z["ss_dim"] + 2 * z["groups"] * z["state"]
        return {"in": ((inner + ch + z["ss_heads"], D), "matrix"), "conv": ((ch, 4), "taps"), "conv.b": ((ch,), "bias"),
                "dt_bias": ((z["ss_heads"],), "step"), "A_log": ((z["ss_heads"],), "rate"), "D": ((z["ss_heads"],), "norm"),
                "norm": ((inner,), "norm"), "o": ((D, inner), "matrix")}
    if kind in ("experts", "experts_shared"):
        E, F = z["experts"], z["expert_ff"]
        names = [f"e{e}." for e in range(E)] + (["shared."] if kind == "experts_shared" else [])
        out = {"router": ((E, D), "matrix")}
        if kind == "experts":
            out["correction"] = ((E,), "bias")
        for n in names:
            if kind == "experts":
                out[n + "gate"] = ((F, D), "matrix")
            out.update({n + "up": ((F, D), "matrix"), n + "down": ((D, F), "matrix")})
        return out
    if kind in ("latent", "latent_low_rank"):
        H, d, r, e, L = z["lat_heads"], z["lat_dim"], z["rot"], z["vdim"], z["kv_rank"]
        out = {"dkv": ((L + r, D), "matrix"), "dkv.norm": ((L,), "norm"), "uk": ((H * d, L), "matrix"), "uv": ((H * e, L), "matrix"),
               "o": ((D, H * e), "matrix")}
        if kind == "latent":
            return dict(out, q=((H * (d + r), D), "matrix"), g=((H, D), "matrix"))
        return dict(out, **{"dq": ((z["q_rank"], D), "matrix"), "dq.norm": ((z["q_rank"],), "norm"),
                            "uq": ((H * (d + r), z["q_rank"]), "matrix"), "sink": ((H,), "bias")})
    if kind == "delta":
        H, G = z["d_heads"], z["d_kv"]
        return {"q": ((G * 128, D), "matrix"), "k": ((G * 128, D), "matrix"), "v": ((H * 128, D), "matrix"), "q.conv": ((G * 128, 4), "taps"),
                "k.conv": ((G * 128, 4), "taps"), "v.conv": ((H * 128, 4), "taps"), "b": ((H, D), "matrix"), "a": ((H, D), "matrix"),
                "A_log": ((H,), "rate"), "dt_bias": ((H,), "step"), "g": ((H * 128, D), "matrix"), "norm": ((128,), "norm"),
                "o": ((D, H * 128), "matrix")}
    if kind == "gla":
        n = z["lat_heads"] * 128
        return {"q": ((n, D), "matrix"), "k": ((n, D), "matrix"), "v": ((n, D), "matrix"), "g": ((n, D), "matrix"),
                "a1": ((z["rank"], D), "matrix"), "a2": ((n, z["rank"]), "matrix"), "a2.b": ((n,), "bias"), "norm": ((128,), "norm"),
                "o": ((D, n), "matrix")}
    if kind == "diff":
        H, G = z["heads"], z["kv"]
        out = {"q": ((H * 128, D), "matrix"), "k": ((G * 128, D), "matrix"), "v": ((G * 128, D), "matrix"), "g": ((H * 128, D), "matrix"),
               "o": ((D, H * 128), "matrix")}
        out.update({n: ((64,), "vector") for n in ("lq1", "lk1", "lq2", "lk2")})
        return out
    raise ValueError(f"unknown kind {kind!r}")


# -- inputs, from the seed alone --------------------------------------------------------------------------------------
def tensor(gen, shape, how):
    def normal():
        return torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32)

    def even(lo, hi):
        return torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float32) * (hi - lo) + lo

    if how == "matrix":
        return (normal() * shape[-1] ** -0.5).to(torch.bfloat16)
    if how == "table":
        return (normal() * 0.02).to(torch.bfloat16)
    if how == "norm":
        return 1.0 + even(-0.1, 0.1)
    if how == "taps":
        return normal() * shape[-1] ** -0.5
    if how == "rate":                            # decay rates of 1 to 16 for a step of one
        return torch.log(even(1.0, 16.0))
    if how == "step":                            # softplus of it: steps of 0.001 to 0.1
        return torch.log(torch.expm1(torch.exp(even(math.log(1e-3), math.log(0.1)))))
    if how == "vector":
        return normal() * (0.5 / shape[0] ** 0.5)
    return normal() * 0.02


def inputs(case, seed):
    """(tensors by name, the step's rows [T, width] or tokens, the rows or tokens before them per request, recurrent state)."""
    gen = torch.Generator(device=DEVICE).manual_seed(1000003 * seed + 17)
    w = {n: tensor(gen, shape, how) for n, (shape, how) in tensor_shapes(case).items()}
    T, kind = case["tokens"], case["kind"]
    if kind == "step":
        vocab = QWEN3[case["size"]]["vocab"]
        x = torch.randint(0, vocab, (T,), generator=gen, device=DEVICE)
        return w, x, [torch.randint(0, vocab, (c,), generator=gen, device=DEVICE) for c in contexts(case)], None
    width = QWEN3[case["size"]]["hidden"] if case["size"] == "4b" else SIZES[case["size"]]["width"]

    def rows(n):
        return torch.randn((n, width), generator=gen, device=DEVICE, dtype=torch.float32).to(torch.bfloat16)

    x = rows(T)
    before = [rows(c) for c in contexts(case)] if case["context"] else []
    state = None
    if kind in ("state_space", "delta", "gla"):
        z, R = SIZES[case["size"]], case["requests"]
        if kind == "state_space":
            shape, ch = (R, z["ss_heads"], z["state"], z["ss_dim"]), z["ss_heads"] * z["ss_dim"] + 2 * z["groups"] * z["state"]
        else:
            shape, ch = (R, z["d_heads"] if kind == "delta" else z["lat_heads"], 128, 128), (2 * z["d_kv"] + z["d_heads"]) * 128
        state = [0.1 * torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32)]
        if kind != "gla":                        # the last inputs of the convolution over four tokens
            state.append(torch.randn((R, 3, ch), generator=gen, device=DEVICE, dtype=torch.float32).to(torch.bfloat16))
    return w, x, before, state


# -- the calls --------------------------------------------------------------------------------------------------------
class Step:
    """What a program keeps between calls: ``call()`` runs the step and returns its outputs.  A recorded step reads the
    weights, the cache and the batch where they lay when it was recorded: ``keep`` holds what owns them."""

    def __init__(self, call, keep=()):
        self.call, self.keep = call, keep


def prepare_step(case, seed):
    """The whole model through the runner: prompts first, then the captured decode step."""
    from prelude_b200.config import load_model_config
    from prelude_b200.engine.graph import DecodeGraphs
    from prelude_b200.engine.loading import build_model, make_runner
    from prelude_b200.engine.runner import StepEntry
    from prelude_b200.weights.loader import WeightStore
    w, x, before, _ = inputs(case, seed)
    model = build_model(load_model_config(qwen3_config(QWEN3[case["size"]])).to_model_spec(), WeightStore.from_tensors(w), "bf16", DEVICE)
    del w
    lens = contexts(case)
    longest = max(lens) + PAGE
    runner = make_runner(model, page_size=PAGE, num_pages=sum(-(-(c + 1) // PAGE) for c in lens) + 1, max_slots=case["requests"],
                         max_request_tokens=longest)
    for r, tokens in enumerate(before):
        runner.step([StepEntry(r, tokens.tolist(), [])])
    for r, c in enumerate(lens):
        runner.cache.grow(r, c + 1)              # room for the token of the decode step
    runner.cache.flush_table_updates()
    graph = DecodeGraphs(runner, 64).get(case["requests"])
    R = case["requests"]
    load = (x.tolist(), lens, [runner.cache.slot_of(r) for r in range(R)], [0.0] * R, [0] * R, [0] * R)
    graph.load(*load)
    graph.capture()

    def call():
        graph.load(*load)
        graph.replay()
        return {"logits": graph.logits}
    return Step(call, (runner, graph))


def prepare(case, seed):
    from prelude_b200.cache.manager import CacheManager
    from prelude_b200.config import load_model_config
    from prelude_b200.engine.batch import StepItem, build_step_batch
    from prelude_b200.engine.capture import no_collection
    from prelude_b200.ops.linear import step_status
    from prelude_b200.parts import model as _registers_the_parts  # noqa: F401
    from prelude_b200.parts.registry import RunContext, make_part
    if case["kind"] == "step":
        return prepare_step(case, seed)
    device = torch.device(DEVICE)
    w, x, before, state = inputs(case, seed)
    config, which = config_of(case)
    block = load_model_config(config).to_model_spec().blocks[0]
    if which == "feed_forward":
        part = make_part("feed_forward", block.feed_forward, "m")
    else:
        part = make_part("mixer", block.mixer.mixers[1] if which == "mixer.1" else block.mixer, "m")
    part.load(lambda name: w[name[2:]], RunContext(device, torch.bfloat16))
    del w
    T, lens, past = case["tokens"], portions(case), contexts(case)
    if which == "feed_forward":
        def forward():
            y = part.forward(x)
            return {"y": y.materialize() if hasattr(y, "materialize") else y}
        captured = T <= CAPTURED_TOKENS
    else:
        R = case["requests"]
        pages = sum(-(-(c + n) // PAGE) for c, n in zip(past, lens)) + 1
        cache = CacheManager([part.cache_need()], PAGE, pages, R, device, torch.bfloat16)
        mine = cache.layer_cache(0)

        def batch_of(items):
            rids = [i.request_id for i in items]
            return build_step_batch(items, cache.block_tables(rids), [cache.slot_of(r) for r in rids], device, 2, 1 << 20)

        for r in range(R):
            cache.add_request(r)
            cache.grow(r, past[r] + lens[r])
        cache.zero_fresh_state()
        for r, rows in enumerate(before):
            b = batch_of([StepItem(r, [0] * past[r], 0)])
            with step_status(b.status):
                part.forward(rows, b, mine)
        held = []
        if state is not None:
            held = [mine.state] if case["kind"] == "gla" else [c.state for c in mine.children]
            slots = torch.tensor([cache.slot_of(r) for r in range(R)], device=device)
            for t, s in zip(held, state):
                t.index_copy_(0, slots, s)
        batch = batch_of([StepItem(r, [0] * n, c) for r, (n, c) in enumerate(zip(lens, past))])
        captured = case["mode"] == "decode" or (T <= CAPTURED_TOKENS and state is not None)

        def forward():
            with step_status(batch.status):
                return {"y": part.forward(x, batch, mine), **{f"state{i}": t for i, t in enumerate(held)}}
    if not captured:
        return Step(forward)
    # as the engine captures a step: once for real, then recorded; what the recurrences moved is put back
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        forward()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    if which != "feed_forward" and state is not None:
        for t, s in zip(held, state):
            t.index_copy_(0, slots, s)
    graph = torch.cuda.CUDAGraph()
    with no_collection(), torch.cuda.graph(graph):
        out = forward()

    def replay():
        graph.replay()
        return out
    return Step(replay, (graph, forward, out))


def run(state):
    return state.call()


# -- what a pass cannot do without ------------------------------------------------------------------------------------
def work(case):
    """Weights once (of routed experts those that are expected to be hit), rows in and out once, what the cache holds of the
    requests once, recurrent state in and out; products of the layer's own formulas."""
    kind, T = case["kind"], case["tokens"]
    shapes = {n: s for n, (s, how) in tensor_shapes(case).items()}
    weights = {n: 2 * math.prod(s) for n, s in shapes.items()}
    keys = [(c, n) for c, n in zip(contexts(case), portions(case))]
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in keys)            # query-key pairs that the causal mask leaves
    cached = sum(c + n for c, n in keys)
    dense = sum(2 * math.prod(s) for s in shapes.values() if len(s) == 2 and s[1] > 8)
    if kind == "step":
        z = QWEN3[case["size"]]
        kv = z["layers"] * 2 * z["kv"] * z["dim"] * 2
        return {"bytes": sum(weights.values()) + cached * kv + T * z["vocab"] * 4,
                "flops": T * dense + z["layers"] * 4 * z["heads"] * z["dim"] * pairs}
    width = next(s for s in shapes.values() if len(s) == 2 and s[1] > 8)[1]
    if case["size"] != "4b":
        width = SIZES[case["size"]]["width"]
    rows = 2 * T * width * 2
    if kind == "mlp":
        return {"bytes": sum(weights.values()) + rows, "flops": T * dense}
    if kind == "attention":
        z = QWEN3[case["size"]]
        return {"bytes": sum(weights.values()) + rows + cached * 2 * z["kv"] * z["dim"] * 2,
                "flops": T * dense + 4 * z["heads"] * z["dim"] * pairs}
    z = SIZES[case["size"]]
    if kind in ("experts", "experts_shared"):
        E, k = z["experts"], z["top"]
        hit = E * (1 - (1 - k / E) ** T)
        each = sum(v for n, v in weights.items() if n.startswith("e0."))
        rest = sum(v for n, v in weights.items() if not n.startswith("e"))
        return {"bytes": hit * each + rest + rows, "flops": T * (k * each + rest)}
    if kind in ("latent", "latent_low_rank"):
        per_pair = 2 * (z["kv_rank"] + z["rot"]) + 2 * z["kv_rank"] if case["mode"] == "decode" else 2 * (z["lat_dim"] + z["rot"]) + 2 * z["vdim"]
        return {"bytes": sum(weights.values()) + rows + cached * (z["kv_rank"] + z["rot"]) * 2, "flops": T * dense + z["lat_heads"] * per_pair * pairs}
    if kind == "diff":
        return {"bytes": sum(weights.values()) + rows + cached * z["kv"] * 256 * 2, "flops": T * dense + z["heads"] * 2 * (2 * 64 + 2 * 128) * pairs}
    held = case["requests"] * {"state_space": z["ss_heads"] * z["state"] * z["ss_dim"], "delta": z["d_heads"] * 128 * 128,
                               "gla": z["lat_heads"] * 128 * 128}[kind]
    each = {"state_space": 6, "delta": 9, "gla": 5}[kind]             # operations an element of the state and token
    return {"bytes": sum(weights.values()) + rows + 2 * 4 * held, "flops": T * dense + each * T * (held // case["requests"])}


def tolerance(case):
    """Roundings to bfloat16 between a layer's kernels; a whole model passes through four layers of them."""
    return {"rel": 2e-2 if case["kind"] == "step" else 1e-2, "max": 0.2}


# -- the same in 64 bits ----------------------------------------------------------------------------------------------
def rms(x, weight, eps=EPS):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def silu(x):
    return x * torch.sigmoid(x)


def turn(x, positions, rates, amplitude, adjacent):
    """x [n, heads, d]: rate i turns entries 2i and 2i + 1 (``adjacent``) or i and i + d / 2 by position * rate."""
    ang = positions.double().view(-1, 1, 1) * rates.view(1, 1, -1)
    c, s, n = ang.cos() * amplitude, ang.sin() * amplitude, rates.numel()
    a, b = (x[..., 0::2], x[..., 1::2]) if adjacent else (x[..., :n], x[..., n:])
    pair = (a * c - b * s, b * c + a * s)
    return torch.stack(pair, -1).flatten(-2) if adjacent else torch.cat(pair, -1)


def plain_rates(dims, base):
    return base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)


def ramped_rates(dims, rot):
    """(rates, amplitude) with long wavelengths slowed down by a factor along a ramp over the pairs."""
    sc, f = rot["scaling"], plain_rates(dims, rot["base"])
    lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[n])) / (2 * math.log(rot["base"])) for n in ("fast", "slow"))
    lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
    ramp = ((torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0


def attend(q, k, v, scale, first, sink=None):
    """q [n, H, d] at positions ``first`` .., k [m, G, d], v [m, G, e] from position 0: causal softmax attention, [n, H, e]."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    ahead = torch.arange(k.shape[0], device=DEVICE).view(1, -1) > torch.arange(first, first + n, device=DEVICE).view(-1, 1)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill(ahead, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out.append(torch.softmax(s, -1)[:, :k.shape[0]] @ v[:, h * G // H])
    return torch.stack(out, 1)


def qwen3_attention(h, w, z, n):
    """h [m, width]: the layer's normed input of one request from position 0; the output of its last ``n`` tokens."""
    m = h.shape[0]
    pos = torch.arange(m, device=DEVICE)
    rates = plain_rates(z["dim"], z["theta"])
    q = turn(rms((h[-n:] @ w["q_proj.weight"].T).view(n, z["heads"], z["dim"]), w["q_norm.weight"]), pos[-n:], rates, 1.0, False)
    k = turn(rms((h @ w["k_proj.weight"].T).view(m, z["kv"], z["dim"]), w["k_norm.weight"]), pos, rates, 1.0, False)
    v = (h @ w["v_proj.weight"].T).view(m, z["kv"], z["dim"])
    return attend(q, k, v, z["dim"] ** -0.5, m - n).flatten(1) @ w["o_proj.weight"].T


def gated(h, gate, up, down):
    return (silu(h @ gate.T) * (h @ up.T)) @ down.T


def latent(h, w, case, n):
    z, m = SIZES[case["size"]], h.shape[0]
    H, d, r, L = z["lat_heads"], z["lat_dim"], z["rot"], z["kv_rank"]
    pos, low = torch.arange(m, device=DEVICE), case["kind"] == "latent_low_rank"
    rates, amplitude = ramped_rates(r, LOW_RANK_ROT) if low else (plain_rates(r, 100000.0), 1.0)
    q = (rms(h[-n:] @ w["dq"].T, w["dq.norm"]) @ w["uq"].T if low else h[-n:] @ w["q"].T).view(n, H, d + r)
    y = h @ w["dkv"].T
    c = rms(y[:, :L], w["dkv.norm"])
    q = torch.cat([q[..., :d], turn(q[..., d:], pos[-n:], rates, amplitude, not low)], -1)
    turned = turn(y[:, None, L:], pos, rates, amplitude, not low)
    k = torch.cat([(c @ w["uk"].T).view(m, H, d), turned.expand(m, H, r)], -1)
    o = attend(q, k, (c @ w["uv"].T).view(m, H, z["vdim"]), (d + r) ** -0.5, m - n, w["sink"] if low else None)
    if not low:
        o = o * torch.sigmoid(h[-n:] @ w["g"].T).unsqueeze(-1)
    return o.flatten(1) @ w["o"].T


def differential(h, w, case):
    z, n = SIZES[case["size"]], h.shape[0]
    H, G = z["heads"], z["kv"]
    q, k = (h @ w["q"].T).view(n, H, 2, 64), (h @ w["k"].T).view(n, G, 2, 64)
    v = (h @ w["v"].T).view(n, G, 128)
    q = q * (1 + 0.1 * torch.log(((torch.arange(n, device=DEVICE) + 1) // 512 + 1).double())).view(n, 1, 1, 1)
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + 0.5
    o = attend(q[:, :, 0], k[:, :, 0], v, 64 ** -0.5, 0) - lam * attend(q[:, :, 1], k[:, :, 1], v, 64 ** -0.5, 0)
    return (rms(o, None).flatten(1) * 0.5 * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def convolved(u, carried, taps, bias=None):
    """(SiLU of the causal convolution over four tokens of u [n, C] behind the three before it, the last three inputs)."""
    u = torch.cat([carried, u])
    n = u.shape[0] - 3
    out = sum(u[j:j + n] * taps[:, j] for j in range(4))
    return silu(out if bias is None else out + bias), u[-3:]


def state_space(h, w, case, S, carried):
    z, n = SIZES[case["size"]], h.shape[0]
    H, P, N, G = z["ss_heads"], z["ss_dim"], z["state"], z["groups"]
    inner = H * P
    proj = h @ w["in"].T
    u, carried = convolved(proj[:, inner:2 * inner + 2 * G * N], carried, w["conv"], w["conv.b"])
    x = u[:, :inner].view(n, H, P)
    B, C = (u[:, inner + i * G * N:inner + (i + 1) * G * N].view(n, G, N).repeat_interleave(H // G, 1) for i in (0, 1))
    dt = torch.nn.functional.softplus(proj[:, 2 * inner + 2 * G * N:] + w["dt_bias"])
    decay, step, y = torch.exp(-torch.exp(w["A_log"]) * dt), dt.unsqueeze(-1) * x, torch.empty_like(x)
    for t in range(n):
        S = torch.baddbmm(decay[t].view(H, 1, 1) * S, B[t].unsqueeze(2), step[t].unsqueeze(1))
        y[t] = torch.bmm(C[t].unsqueeze(1), S).squeeze(1)
    y = (y + w["D"].view(H, 1) * x).reshape(n, inner) * silu(proj[:, :inner])
    return (rms(y.view(n, z["groups"], -1), None).reshape(n, inner) * w["norm"]) @ w["o"].T, S, carried


def delta_rule(h, w, case, S, carried):
    z, n = SIZES[case["size"]], h.shape[0]
    H, G = z["d_heads"], z["d_kv"]
    u, carried = convolved(h @ torch.cat([w["q"], w["k"], w["v"]]).T, carried, torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]))
    q, k, v = u[:, :G * 128].view(n, G, 128), u[:, G * 128:2 * G * 128].view(n, G, 128), u[:, 2 * G * 128:].view(n, H, 128)
    q, k = ((t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1) for t in (q, k))
    q = q * 128 ** -0.5
    beta = torch.sigmoid(h @ w["b"].T)
    decay = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))
    o = torch.empty_like(v)
    for t in range(n):
        S = decay[t].view(H, 1, 1) * S
        d = beta[t].view(H, 1, 1) * (v[t].unsqueeze(1) - torch.bmm(k[t].unsqueeze(1), S))
        S = torch.baddbmm(S, k[t].unsqueeze(2), d)
        o[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
    o = rms(o, w["norm"]).flatten(1) * silu(h @ w["g"].T)
    return o @ w["o"].T, S, carried


def linear_attention(h, w, case, S):
    H, n = SIZES[case["size"]]["lat_heads"], h.shape[0]
    q, k, v = ((h @ w[c].T).view(n, H, 128) for c in "qkv")
    q = q * 128 ** -0.5
    a = torch.exp(torch.nn.functional.logsigmoid((h @ w["a1"].T) @ w["a2"].T + w["a2.b"]) / 16.0).view(n, H, 128)
    o = torch.empty_like(v)
    for t in range(n):
        S = torch.baddbmm(a[t].unsqueeze(2) * S, k[t].unsqueeze(2), v[t].unsqueeze(1))
        o[t] = torch.bmm(q[t].unsqueeze(1), S).squeeze(1)
    return (rms(o, w["norm"]).flatten(1) * silu(h @ w["g"].T)) @ w["o"].T, S


def routed(h, w, case):
    z, shared = SIZES[case["size"]], case["kind"] == "experts_shared"
    E, k = z["experts"], z["top"]
    logits = h @ w["router"].double().T
    score = torch.softmax(logits, -1) if shared else torch.sigmoid(logits)
    choice = score if shared else score + w["correction"].double()
    groups = choice.view(-1, 4, E // 4)
    best = (groups.amax(-1) if shared else groups.topk(2, -1).values.sum(-1)).topk(2, -1).indices
    kept = torch.zeros(h.shape[0], 4, dtype=torch.bool, device=DEVICE).scatter_(1, best, True).repeat_interleave(E // 4, 1)
    ids = choice.masked_fill(~kept, -math.inf).topk(k, -1).indices
    p = score.gather(1, ids)
    if shared:
        p = p / (p.sum(-1, keepdim=True) + 1e-20) * 1.5

    def expert(x, name):
        m = {n: w[f"{name}.{n}"].double() for n in (("up", "down") if shared else ("gate", "up", "down"))}
        return torch.relu(x @ m["up"].T) ** 2 @ m["down"].T if shared else gated(x, m["gate"], m["up"], m["down"])

    out = expert(h, "shared") if shared else torch.zeros_like(h)
    for e in range(E):
        row, slot = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            out.index_add_(0, row, p[row, slot].unsqueeze(1) * expert(h[row], f"e{e}"))
    return out


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    raw, x, before, state = inputs(case, seed)
    if kind in ("experts", "experts_shared"):
        return {"y": routed(x.double(), raw, case)}
    if kind == "step":
        return {"logits": exact_step(case, raw, x, before)}
    w, x = {n: t.double() for n, t in raw.items()}, x.double()
    if kind == "mlp":
        return {"y": gated(x, w["gate_proj.weight"], w["up_proj.weight"], w["down_proj.weight"])}
    out, at = {"y": []}, 0
    ends = [[] for _ in state or ()]
    for r, n in enumerate(portions(case)):
        h, at = x[at:at + n], at + n
        if before:
            h = torch.cat([before[r].double(), h])
        if kind == "attention":
            y = qwen3_attention(h, w, QWEN3[case["size"]], n)
        elif kind in ("latent", "latent_low_rank"):
            y = latent(h, w, case, n)
        elif kind == "diff":
            y = differential(h, w, case)
        else:
            step = {"state_space": state_space, "delta": delta_rule, "gla": linear_attention}[kind]
            y, *moved = step(h, w, case, *(s[r].double() for s in state))
            for e, m in zip(ends, moved):
                e.append(m)
        out["y"].append(y)
    out["y"] = torch.cat(out["y"])
    out.update({f"state{i}": torch.stack(e) for i, e in enumerate(ends)})
    return out


def exact_step(case, raw, x, before):
    """Logits of every request's newest token: the whole model over each request's tokens, layer by layer."""
    z = QWEN3[case["size"]]
    table = raw["model.embed_tokens.weight"]
    streams = [table[torch.cat([b, x[r:r + 1]])].double() for r, b in enumerate(before)]
    for i in range(z["layers"]):
        p = f"model.layers.{i}."
        w = {n[len(p):]: t.double() for n, t in raw.items() if n.startswith(p)}
        att = {n[10:]: t for n, t in w.items() if n.startswith("self_attn.")}
        for r, res in enumerate(streams):
            n = 1 if i == z["layers"] - 1 else res.shape[0]          # of the last layer only the newest token is wanted
            res = res[-n:] + qwen3_attention(rms(res, w["input_layernorm.weight"]), att, z, n)
            streams[r] = res + gated(rms(res, w["post_attention_layernorm.weight"]), w["mlp.gate_proj.weight"], w["mlp.up_proj.weight"],
                                     w["mlp.down_proj.weight"])
    last = rms(torch.cat(streams), raw["model.norm.weight"].double())
    return torch.cat([last @ part.double().T for part in table.split(16384)], 1)
