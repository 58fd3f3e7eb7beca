"""Timed cases of the generation library: what a program asks of it between a request's tokens and its next token.

Whole decode steps go through `Engine.step` (a captured graph per batch size, as every generation loop uses it); prompts are timed
layer by layer, through the parts that a model is assembled from (`Mixer.forward`, `FeedForward.forward`) on a step's metadata and a
`SequenceCache`.  Model sizes are those of `bench.py`: dense Qwen3 at the 0.6B, 8B and 32B widths, Fasesun and Pegurax layers at the
widths 1,024 to 4,096.  Weights and inputs are random; cached positions are filled with random keys, values and latents.

`exact` states the same results in 64-bit arithmetic from the formulas, with nothing of the library.
"""
import math

import numpy as np
import torch

import tau_rs_b200  # noqa: F401  (registers the parts)
from tau_rs_b200 import DecoderModel, Engine, SequenceCache, StepEntry
from tau_rs_b200.config.registry import architecture_for
from tau_rs_b200.config.specs import DeltaRuleSpec
from tau_rs_b200.engine.batch import StepLayout, fill_step, step_views
from tau_rs_b200.parts import build

PAGE = 64

# hidden, query heads, key/value heads, feed-forward, tied head: the Qwen3 shapes of bench.py
QWEN3 = {"0.6b": (1024, 16, 8, 3072, True), "8b": (4096, 32, 8, 12288, False), "32b": (5120, 64, 8, 25600, False)}
# width -> latent heads, query rank, memory heads, expert width, shared expert's width: the Fasesun sizes of bench.py
FASESUN = {1024: (8, 384, 2, 704, 1408), 2048: (16, 768, 4, 1408, 2816), 4096: (32, 1536, 8, 2048, 4096)}
EXPERTS, TOP = 64, 6


def listed():
    return [
        # One request alone on the small model: a chat turn's next token, where launches and latency count.
        {"name": "qwen3_0.6b_decode_1", "kind": "decode", "shape": "0.6b", "layers": 28, "batch": 1, "context": 300, "ragged": False},
        # The benchmark's decode step: 8 requests of 2,048 tokens at the 8B widths (4 of the 36 layers, the whole head).
        {"name": "qwen3_8b_decode_8", "kind": "decode", "shape": "8b", "layers": 4, "batch": 8, "context": 2048, "ragged": False},
        # A busy server: 64 requests of unequal lengths in one step.
        {"name": "qwen3_8b_decode_64", "kind": "decode", "shape": "8b", "layers": 4, "batch": 64, "context": 1500, "ragged": True},
        # The benchmark's prompt: 2,048 fresh tokens through a layer's attention and feed-forward.
        {"name": "qwen3_8b_prompt_2048", "kind": "layer", "shape": "8b", "sequences": 1, "new": 2048, "cached": 0, "ragged": False, "dtype": "bfloat16"},
        # Portions of several prompts in one step, each continuing what is cached (chunked prefill of unequal requests).
        {"name": "qwen3_8b_portions_ragged", "kind": "layer", "shape": "8b", "sequences": 6, "new": 120, "cached": 1500, "ragged": True, "dtype": "bfloat16"},
        # The true 32-bit run (`--dtype float32`) of a prompt at the 0.6B widths.
        {"name": "qwen3_0.6b_prompt_float32", "kind": "layer", "shape": "0.6b", "sequences": 1, "new": 777, "cached": 0, "ragged": False, "dtype": "float32"},
        # A prompt through latent attention.
        {"name": "latent_prompt_2048", "kind": "latent", "width": 2048, "sequences": 1, "new": 2048},
        # A decode step through four latent-attention layers.
        {"name": "latent_decode_8", "kind": "latent_decode", "width": 2048, "layers": 4, "batch": 8, "context": 2048},
        # A prompt through a matrix memory (mLSTM).
        {"name": "mlstm_prompt_2048", "kind": "memory", "type": "mlstm", "width": 2048, "sequences": 1, "new": 2048},
        # A prompt through the gated delta rule.
        {"name": "delta_prompt_2048", "kind": "delta", "width": 2048, "sequences": 1, "new": 2048},
        # A prompt through routed experts, and a decode step of 8 through them.
        {"name": "experts_prompt_2048", "kind": "experts", "width": 2048, "tokens": 2048, "single": False},
        {"name": "experts_decode_8", "kind": "experts", "width": 2048, "tokens": 8, "single": True},
    ]


def _between(rng, low, high):
    """A whole number between `low` and `high`, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "layer", "layer", "latent", "latent_decode", "memory", "delta", "experts", "experts"])
    width = rng.choice([1024, 2048])
    if kind == "decode":
        shape = rng.choice(["0.6b", "8b"])
        return {"kind": kind, "shape": shape, "layers": 28 if shape == "0.6b" else 4, "batch": _between(rng, 1, 32 if shape == "0.6b" else 64),
                "context": _between(rng, 20, 2000), "ragged": rng.random() < 0.5}
    if kind == "layer":
        shape, dtype = rng.choice([("0.6b", "bfloat16"), ("8b", "bfloat16"), ("8b", "bfloat16"), ("0.6b", "float32")])
        sequences = _between(rng, 1, 8)
        most = (2048 if dtype == "bfloat16" else 768) // sequences
        return {"kind": kind, "shape": shape, "sequences": sequences, "new": _between(rng, 40, most), "cached": rng.choice([0, 0, _between(rng, 30, 2000)]),
                "ragged": rng.random() < 0.7, "dtype": dtype}
    if kind == "latent":
        sequences = _between(rng, 1, 4)
        return {"kind": kind, "width": width, "sequences": sequences, "new": _between(rng, 150, 2048 // sequences)}
    if kind == "latent_decode":
        return {"kind": kind, "width": width, "layers": 4, "batch": _between(rng, 1, 24), "context": _between(rng, 60, 2400)}
    if kind in ("memory", "delta"):
        sequences = _between(rng, 1, 4)
        case = {"kind": kind, "width": width, "sequences": sequences, "new": _between(rng, 100, 2048 // sequences)}
        return {**case, "type": rng.choice(["mlstm", "lightning"])} if kind == "memory" else case
    single = rng.random() < 0.4
    return {"kind": kind, "width": width, "tokens": _between(rng, 1, 32) if single else _between(rng, 100, 2048), "single": single}


# ---- sizes and weights ------------------------------------------------------------------------------------------------
def _lengths(case):
    """New and cached tokens of each sequence of a step."""
    count, new, cached = case.get("sequences", 1), case["new"], case.get("cached", 0)
    if not case.get("ragged"):
        return [new] * count, [cached] * count
    return [max(2, new - (new * i * 3) // (4 * count)) for i in range(count)], [cached * (count - i) // count for i in range(count)]


def _contexts(case):
    count, context = case["batch"], case["context"]
    return [max(1, context - (context * i * 3) // (4 * count)) if case.get("ragged") else context for i in range(count)]


def _qwen3_config(case, layers):
    hidden, heads, kv_heads, intermediate, tied = QWEN3[case["shape"]]
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": layers, "hidden_size": hidden, "num_attention_heads": heads,
            "num_key_value_heads": kv_heads, "head_dim": 128, "intermediate_size": intermediate, "vocab_size": 151936 if case["kind"] == "decode" else 64,
            "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": tied, "attention_bias": False, "max_position_embeddings": 40960,
            "hidden_act": "silu", "torch_dtype": case.get("dtype", "bfloat16")}


def _decays(heads):
    return [1.0 - 2.0 ** (-5 - 3 * h / heads) for h in range(heads)]


def _fasesun_config(case):
    width = case["width"]
    heads, q_rank, memory_heads, expert_ff, shared_ff = FASESUN[width]
    latent = {"type": "latent_attention", "mlp": None,
              "mixer": {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": q_rank, "kv_rank": 512, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}}
    if case["kind"] == "memory":
        if case["type"] == "mlstm":
            layer = {"type": "mlstm", "mlp": None, "mixer": {"heads": memory_heads, "dim": 256, "vdim": 512, "gate_cap": 15.0}}
        else:
            layer = {"type": "lightning", "mlp": None, "mixer": {"heads": heads, "dim": 128, "vdim": 128, "decay": _decays(heads)}}
    elif case["kind"] == "experts":
        layer = dict(latent, mlp={"kind": "moe", "router": {"experts": EXPERTS, "top": TOP}, "expert": {"ff": expert_ff}, "shared": {"ff": shared_ff}})
    else:
        layer = latent
    layers = [layer] * case.get("layers", 1)
    return {"architecture": "Fasesun", "layers": layers, "norm": {"eps": 1e-5}, "vocab": 32768 if case["kind"] == "latent_decode" else 64, "width": width}


def _delta_sizes(case):
    heads = case["width"] // 128
    return heads, heads // 2, 128, 128, 4      # heads, key heads, key width, value width, taps


def _shapes(case):
    """Tensor name -> (shape, how its values are drawn): the parts of a layer that the case runs."""
    kind = case["kind"]
    if kind in ("decode", "layer"):
        hidden, heads, kv_heads, inner, tied = QWEN3[case["shape"]]
        vocab = 151936 if kind == "decode" else 64
        out = {"model.embed_tokens.weight": ((vocab, hidden), "matrix")}
        for i in range(case.get("layers", 1)):
            p = f"model.layers.{i}."
            out.update({p + "input_layernorm.weight": ((hidden,), "ones"), p + "self_attn.q_proj.weight": ((heads * 128, hidden), "matrix"),
                        p + "self_attn.k_proj.weight": ((kv_heads * 128, hidden), "matrix"), p + "self_attn.v_proj.weight": ((kv_heads * 128, hidden), "matrix"),
                        p + "self_attn.o_proj.weight": ((hidden, heads * 128), "matrix"), p + "self_attn.q_norm.weight": ((128,), "ones"),
                        p + "self_attn.k_norm.weight": ((128,), "ones"), p + "post_attention_layernorm.weight": ((hidden,), "ones"),
                        p + "mlp.gate_proj.weight": ((inner, hidden), "matrix"), p + "mlp.up_proj.weight": ((inner, hidden), "matrix"),
                        p + "mlp.down_proj.weight": ((hidden, inner), "matrix")})
        out["model.norm.weight"] = ((hidden,), "ones")
        if not tied:
            out["lm_head.weight"] = ((vocab, hidden), "matrix")
        return out
    width = case["width"]
    if kind == "delta":
        heads, key_heads, dim, vdim, taps = _delta_sizes(case)
        k, v = key_heads * dim, heads * vdim
        return {"m.q": ((k, width), "matrix"), "m.k": ((k, width), "matrix"), "m.v": ((v, width), "matrix"), "m.g": ((v, width), "matrix"),
                "m.b": ((heads, width), "matrix"), "m.a": ((heads, width), "matrix"), "m.o": ((width, v), "matrix"), "m.q.conv": ((k, taps), "taps"),
                "m.k.conv": ((k, taps), "taps"), "m.v.conv": ((v, taps), "taps"), "m.A_log": ((heads,), "rates"), "m.dt_bias": ((heads,), "steps"),
                "m.norm": ((vdim,), "ones")}
    heads, q_rank, memory_heads, expert_ff, shared_ff = FASESUN[width]
    out = {"embed": ((32768 if kind == "latent_decode" else 64, width), "matrix"), "final.norm": ((width,), "ones")}
    for i in range(case.get("layers", 1)):
        out[f"l{i}.norm1"] = ((width,), "ones")
        p = f"l{i}.mix."
        if kind == "memory":
            n, dim, vdim = (memory_heads, 256, 512) if case["type"] == "mlstm" else (heads, 128, 128)
            out.update({p + "q": ((n * dim, width), "matrix"), p + "k": ((n * dim, width), "matrix"), p + "v": ((n * vdim, width), "matrix"),
                        p + "g": ((n * vdim, width), "matrix"), p + "o": ((width, n * vdim), "matrix"), p + "norm": ((n * vdim,), "ones")})
            if case["type"] == "mlstm":
                out.update({p + "i": ((n, width), "matrix"), p + "f": ((n, width), "matrix"), p + "i.b": ((n,), "small"), p + "f.b": ((n,), "remember")})
        else:
            out.update({p + "dq": ((q_rank, width), "matrix"), p + "dq.norm": ((q_rank,), "ones"), p + "uq": ((heads * 192, q_rank), "matrix"),
                        p + "dkv": ((576, width), "matrix"), p + "dkv.norm": ((512,), "ones"), p + "uk": ((heads * 128, 512), "wide"),
                        p + "uv": ((heads * 128, 512), "wide"), p + "sink": ((heads,), "ones"), p + "g": ((heads * 128, width), "matrix"),
                        p + "o": ((width, heads * 128), "matrix")})
        if kind == "experts":
            p = f"l{i}.mlp."
            out.update({p + "router": ((EXPERTS, width), "matrix"), p + "correction": ((EXPERTS,), "small"), p + "shared.sg": ((1, width), "matrix")})
            for name, inner in [("shared", shared_ff)] + [(f"e{e}", expert_ff) for e in range(EXPERTS)]:
                out.update({f"{p}{name}.gate": ((inner, width), "matrix"), f"{p}{name}.up": ((inner, width), "matrix"), f"{p}{name}.down": ((width, inner), "matrix")})
    return out


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _weights(case, generator):
    """Random tensors as a folder of bfloat16 weights holds them (a float32 run widens them); vectors are 32-bit."""
    out = {}
    for name, (shape, how) in _shapes(case).items():
        values = torch.randn(shape, generator=generator, device="cuda", dtype=torch.bfloat16)
        if how == "matrix":
            out[name] = values.mul_(0.02).to(_dtype(case))
        elif how == "wide":
            out[name] = values.mul_(0.04).to(_dtype(case))
        else:
            values = values.float()
            out[name] = {"ones": lambda v: 1.0 + 0.1 * v, "taps": lambda v: 0.3 * v, "small": lambda v: 0.1 * v, "remember": lambda v: 3.0 + 0.5 * v,
                         "rates": lambda v: 1.0 + 0.5 * v, "steps": lambda v: -4.0 + v}[how](values)
    return out


def _spec_dtype(name, value, specs):
    return value.float() if specs[name].role == "vector" else value


def _model(case, config, weights):
    entry = architecture_for(config)
    model = DecoderModel(entry.build_spec(entry.parse_config(config)), _dtype(case), torch.device("cuda:0"))
    specs = model.tensor_specs()
    for name in specs:
        if name not in weights:      # a part that the case does not run
            weights[name] = torch.zeros(specs[name].shape, dtype=_dtype(case), device="cuda")
        model.assign(name, _spec_dtype(name, weights[name], specs))
    model.finalize_weights()
    return model


def _hidden(case, tokens, width, generator):
    return torch.randn((tokens, width), generator=generator, device="cuda", dtype=torch.bfloat16).to(_dtype(case))


def _step(cache, slots, new, cached):
    """The metadata of a step in which sequence i brings `new[i]` tokens behind `cached[i]` positions."""
    for slot, n, c in zip(slots, new, cached):
        cache.reserve(slot, c + n)
    longest = max(n + c for n, c in zip(new, cached))
    layout = StepLayout(sum(new), len(new), 0, {group: -(-longest // PAGE) for group in cache.kv})
    staged = np.zeros(layout.total, dtype=np.int32)
    fill_step(layout, staged, [StepEntry(slot, [0] * n, []) for slot, n in zip(slots, new)], cached, cache)
    step = step_views(layout, torch.from_numpy(staged).cuda(), max(new), longest, all(n == 1 for n in new))
    step.all_fresh = not any(cached)
    for slot, n, c in zip(slots, new, cached):
        cache.advance(slot, c + n)
    return step


def _cached_rows(generator, length, *shape):
    return torch.randn((length, *shape), generator=generator, device="cuda", dtype=torch.bfloat16)


def _fill(pages, table, rows):
    """Cached rows `[length, ...]` into the pages of a sequence (`pages` [pages, ..., 64, d] or [pages, 64, d])."""
    count = -(-rows.shape[0] // PAGE)
    padded = torch.zeros((count * PAGE, *rows.shape[1:]), dtype=pages.dtype, device="cuda")
    padded[: rows.shape[0]] = rows
    padded = padded.view(count, PAGE, *rows.shape[1:])
    numbers = torch.from_numpy(np.ascontiguousarray(table[:count])).long().cuda()
    pages[numbers] = padded.transpose(1, 2) if padded.dim() == 4 else padded


# ---- what a program has in hand, and one pass -------------------------------------------------------------------------
def prepare(case, seed):
    generator = _generator(seed)
    weights = _weights(case, generator)
    kind = case["kind"]
    if kind in ("decode", "latent_decode"):
        model = _model(case, _qwen3_config(case, case["layers"]) if kind == "decode" else _fasesun_config(case), weights)
        contexts = _contexts(case)
        room = 4096 if case["batch"] <= 24 else 2048      # every pass makes the sequences one token longer
        engine = Engine(model, sum(-(-(c + room) // PAGE) * PAGE for c in contexts), max(contexts) + room, max_slots=case["batch"])
        slots = [engine.open_sequence() for _ in contexts]
        (group,) = engine.cache.kv
        for slot, length in zip(slots, contexts):
            engine.cache.reserve(slot, length)
            engine.cache.advance(slot, length)
        for layer in range(case["layers"]):
            view = engine.cache.layer_view(group, layer)
            for slot, length in zip(slots, contexts):
                table = engine.cache.page_rows(group, [slot], engine.cache.pages_per_sequence)[0]
                if kind == "decode":
                    _fill(view.keys, table, _cached_rows(generator, length, QWEN3[case["shape"]][2], 128))
                    _fill(view.values, table, _cached_rows(generator, length, QWEN3[case["shape"]][2], 128))
                else:
                    _fill(view.rows, table, _cached_rows(generator, length, 576))
        tokens = torch.randint(0, 32768, (case["batch"],), generator=generator, device="cuda").tolist()
        return {"kind": kind, "engine": engine, "entries": [StepEntry(slot, [token], (0,)) for slot, token in zip(slots, tokens)]}
    if kind == "experts":
        model = _model(case, _fasesun_config(case), weights)
        slots_cache = SequenceCache(model.cache_groups(), case["tokens"] * PAGE if case["single"] else case["tokens"], 1 << 20, model.dtype, model.device)
        new = [1] * case["tokens"] if case["single"] else [case["tokens"]]
        slots = [slots_cache.open() for _ in new]
        return {"kind": kind, "part": model.blocks[0].feed_forward, "step": _step(slots_cache, slots, new, [0] * len(new)),
                "hidden": _hidden(case, case["tokens"], case["width"], generator)}
    new, cached = _lengths(case)
    positions = sum(-(-(n + c) // PAGE) * PAGE for n, c in zip(new, cached))
    if kind == "delta":
        heads, key_heads, dim, vdim, taps = _delta_sizes(case)
        part = build("mixer", DeltaRuleSpec(hidden=case["width"], n_heads=heads, n_key_heads=key_heads, key_dim=dim, value_dim=vdim, taps=taps, eps=1e-5),
                     prefix="m", dtype=torch.bfloat16, device=torch.device("cuda:0"))
        specs = part.tensor_specs()
        for name in specs:
            part.assign(name, _spec_dtype(name, weights[name], specs))
        part.finalize_weights()
        groups = {"memory": (part.cache_need(), 1), "taps": (part.extra_cache_needs()["taps"], 1)}
        cache = SequenceCache(groups, positions, 1 << 20, torch.bfloat16, torch.device("cuda:0"), max_slots=len(new))
        slots = [cache.open() for _ in new]
        step = _step(cache, slots, new, cached)
        view = cache.layer_view("memory", 0)
        view.extra = {"taps": cache.layer_view("taps", 0)}
        return {"kind": kind, "part": part, "cache": cache, "slots": slots, "step": step, "view": view, "hidden": _hidden(case, sum(new), case["width"], generator)}
    model = _model(case, _qwen3_config(case, 1) if kind == "layer" else _fasesun_config(case), weights)
    cache = SequenceCache(model.cache_groups(), positions, max(n + c for n, c in zip(new, cached)) + PAGE, model.dtype, model.device, max_slots=len(new))
    slots = [cache.open() for _ in new]
    step = _step(cache, slots, new, cached)
    (group,) = model.cache_groups()
    view = cache.layer_view(group, 0)
    state = {"kind": kind, "part": model.blocks[0].mixer, "cache": cache, "slots": slots, "step": step, "view": view}
    if kind == "layer":
        view.keys.zero_()
        view.values.zero_()
        for slot, length in zip(slots, cached):
            table = cache.page_rows(group, [slot], cache.pages_per_sequence)[0]
            _fill(view.keys, table, _cached_rows(generator, length, QWEN3[case["shape"]][2], 128))
            _fill(view.values, table, _cached_rows(generator, length, QWEN3[case["shape"]][2], 128))
        state["mlp"] = model.blocks[0].feed_forward
        width = QWEN3[case["shape"]][0]
        state["second"] = _hidden(case, sum(new), width, generator)
    else:
        width = case["width"]
        if kind == "latent":
            view.rows.zero_()
    state["hidden"] = _hidden(case, sum(new), width, generator)
    return state


def run(state):
    kind = state["kind"]
    if kind in ("decode", "latent_decode"):
        return state["engine"].step(state["entries"])
    if kind == "experts":
        return state["part"].forward(state["hidden"], state["step"])
    view = state["view"]
    if kind in ("memory", "delta"):      # new sequences: their state starts at zero, as a slot is handed out
        for group in state["cache"].states.values():
            group.state.zero_()
        out = state["part"].forward(state["hidden"], state["step"], view, True)
        return [out, view.state] + ([view.extra["taps"].state] if kind == "delta" else [])
    out = state["part"].forward(state["hidden"], state["step"], view, True)
    if kind == "latent":
        return [out, view.rows]
    return [out, state["mlp"].forward(state["second"], state["step"]), view.keys, view.values]


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _product(rows, inputs, outputs, element=2):
    return {"bytes": element * (rows * inputs + inputs * outputs + rows * outputs), "flops": 2 * rows * inputs * outputs}


def _sum(*parts):
    return {"bytes": float(sum(p["bytes"] for p in parts)), "flops": float(sum(p["flops"] for p in parts))}


def _attended(new, cached):
    """(query, key) pairs of causal runs."""
    return sum(n * c + n * (n + 1) // 2 for n, c in zip(new, cached))


def work(case):
    kind = case["kind"]
    if kind == "decode":
        hidden, heads, kv_heads, inner, _ = QWEN3[case["shape"]]
        contexts, b = _contexts(case), case["batch"]
        weights = hidden * (heads + 2 * kv_heads) * 128 + heads * 128 * hidden + 3 * hidden * inner
        keys = sum(c + 1 for c in contexts)
        layer = {"bytes": 2 * weights + 4 * keys * kv_heads * 128, "flops": 2 * b * weights + 4 * keys * heads * 128}
        head = {"bytes": 2 * 151936 * hidden + 4 * b * 151936, "flops": 2 * b * 151936 * hidden}
        return _sum(head, *[layer] * case["layers"])
    if kind == "layer":
        hidden, heads, kv_heads, inner, _ = QWEN3[case["shape"]]
        new, cached = _lengths(case)
        rows, element = sum(new), 4 if case["dtype"] == "float32" else 2
        attention = {"bytes": 2 * element * (sum(new) + sum(cached)) * kv_heads * 128, "flops": 4 * _attended(new, cached) * heads * 128}
        weights = hidden * (heads + 2 * kv_heads) * 128 + heads * 128 * hidden + 3 * hidden * inner
        return _sum(attention, {"bytes": element * (weights + 4 * rows * hidden), "flops": 2 * rows * weights})
    width = case["width"]
    if kind == "delta":
        heads, key_heads, dim, vdim, taps = _delta_sizes(case)
        new, _ = _lengths(case)
        rows = sum(new)
        weights = width * (2 * key_heads * dim + 3 * heads * vdim + 2 * heads)
        state = heads * dim * vdim * len(new)
        return _sum({"bytes": 2 * (weights + 2 * rows * width) + 4 * state, "flops": 2 * rows * weights + 8 * rows * heads * dim * vdim})
    heads, q_rank, memory_heads, expert_ff, shared_ff = FASESUN[width]
    if kind == "memory":
        new, _ = _lengths(case)
        rows = sum(new)
        n, dim, vdim = (memory_heads, 256, 512) if case["type"] == "mlstm" else (heads, 128, 128)
        weights = width * n * (2 * dim + 3 * vdim)
        return _sum({"bytes": 2 * (weights + 2 * rows * width) + 4 * len(new) * n * dim * vdim, "flops": 2 * rows * weights + 5 * rows * n * dim * vdim})
    if kind == "experts":
        rows = case["tokens"]
        touched = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** rows)
        bytes_ = 2 * 3 * width * (touched * expert_ff + shared_ff) + 4 * EXPERTS * width + 2 * rows * width + 4 * rows * width
        return {"bytes": float(bytes_), "flops": float(2 * rows * width * (3 * (TOP * expert_ff + shared_ff) + EXPERTS))}
    weights = width * q_rank + q_rank * heads * 192 + width * 576 + 2 * heads * 128 * 512 + 2 * width * heads * 128
    if kind == "latent":
        new, cached = _lengths(case)
        rows = sum(new)
        return _sum({"bytes": 2 * (weights + 2 * rows * width + rows * 576), "flops": 2 * rows * weights + 2 * _attended(new, cached) * heads * 320})
    contexts, b = _contexts(case), case["batch"]
    keys = sum(c + 1 for c in contexts)
    layer = {"bytes": 2 * weights + 2 * keys * 576, "flops": 2 * b * weights + 2 * keys * heads * (576 + 512)}
    head = {"bytes": 2 * 32768 * width + 4 * b * 32768, "flops": 2 * b * 32768 * width}
    return _sum(head, *[layer] * case["layers"])


def tolerance(case):
    """About four times what this precision shows against 64 bits: 1e-6 in 32-bit sums, 5e-3 for one layer's bfloat16 roundings."""
    if case.get("dtype") == "float32":
        return {"rel": 5e-6}
    if case["kind"] == "decode":                  # a rounding of one layer travels through all that follow: 0.015 over 4 layers, 0.035 over 28
        return {"rel": 0.05 if case["layers"] <= 8 else 0.12}
    return {"rel": 2e-2}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------
def _rms(x, weight, eps):
    x = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return x if weight is None else x * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _half_rotation(x, positions, theta=1000000.0):
    """Element j with j + d/2; the angle is a 32-bit number by the model's definition."""
    d = x.shape[-1]
    inverse = 1.0 / torch.tensor([theta ** (i / d) for i in range(0, d, 2)], dtype=torch.float32, device=x.device)
    angle = (positions.float()[:, None] * inverse[None, :]).double()[:, None, :]
    u, v = x[..., : d // 2], x[..., d // 2 :]
    return torch.cat([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], dim=-1)


def _pair_rotation(x, positions, base=10000.0):
    d = x.shape[-1]
    frequency = torch.tensor([base ** (-2.0 * i / d) for i in range(d // 2)], dtype=torch.float64, device=x.device).float()
    angle = (positions.float()[:, None] * frequency[None, :]).double()
    angle = angle.view(x.shape[0], *[1] * (x.dim() - 2), d // 2)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], dim=-1).flatten(-2)


def _causal_softmax(q, k, v, scale, sink=None):
    """q [n, heads, d], k [m, heads, d], v [m, heads, e]; the queries are the last n of the m positions."""
    n, m = q.shape[0], k.shape[0]
    hidden = torch.arange(m, device=q.device)[None, :] > torch.arange(m - n, m, device=q.device)[:, None]
    out = []
    for h in range(q.shape[1]):
        scores = (q[:, h] @ k[:, h].T * scale).masked_fill(hidden, float("-inf"))
        if sink is not None:
            scores = torch.cat([scores, sink[h].expand(n, 1)], dim=1)
        out.append(torch.softmax(scores, dim=-1)[:, :m] @ v[:, h])
    return torch.stack(out, dim=1)


def _qwen3_attention(h, W, p, case, keys, values, start):
    _, heads, kv_heads, _, _ = QWEN3[case["shape"]]
    n = h.shape[0]
    positions = torch.arange(start, start + n, device=h.device)
    q = _half_rotation(_rms((h @ W[p + "self_attn.q_proj.weight"].T).view(n, heads, 128), W[p + "self_attn.q_norm.weight"], 1e-6), positions)
    k = _half_rotation(_rms((h @ W[p + "self_attn.k_proj.weight"].T).view(n, kv_heads, 128), W[p + "self_attn.k_norm.weight"], 1e-6), positions)
    v = (h @ W[p + "self_attn.v_proj.weight"].T).view(n, kv_heads, 128)
    k, v = torch.cat([keys, k]).repeat_interleave(heads // kv_heads, dim=1), torch.cat([values, v]).repeat_interleave(heads // kv_heads, dim=1)
    return _causal_softmax(q, k, v, 128 ** -0.5).reshape(n, -1) @ W[p + "self_attn.o_proj.weight"].T


def _qwen3_mlp(h, W, p):
    return (_silu(h @ W[p + "mlp.gate_proj.weight"].T) * (h @ W[p + "mlp.up_proj.weight"].T)) @ W[p + "mlp.down_proj.weight"].T


def _latent(h, W, p, heads, latents, start):
    """`latents` [cached, 576]: normalised latents and rotated key parts; returns the result and the rows that join them."""
    n = h.shape[0]
    positions = torch.arange(start, start + n, device=h.device)
    q = (_rms(h @ W[p + "dq"].T, W[p + "dq.norm"], 1e-5) @ W[p + "uq"].T).view(n, heads, 192)
    down = h @ W[p + "dkv"].T
    rows = torch.cat([_rms(down[:, :512], W[p + "dkv.norm"], 1e-5), _pair_rotation(down[:, 512:], positions)], dim=1)
    every = torch.cat([latents, rows])
    m = every.shape[0]
    k = torch.cat([(every[:, :512] @ W[p + "uk"].T).view(m, heads, 128), every[:, None, 512:].expand(m, heads, 64)], dim=-1)
    q = torch.cat([q[..., :128], _pair_rotation(q[..., 128:], positions)], dim=-1)
    mixed = _causal_softmax(q, k, (every[:, :512] @ W[p + "uv"].T).view(m, heads, 128), 192 ** -0.5, W[p + "sink"]).reshape(n, -1)
    return (mixed * torch.sigmoid(h @ W[p + "g"].T)) @ W[p + "o"].T, rows


def _memory(h, W, p, case, new):
    heads, _, memory_heads, _, _ = FASESUN[case["width"]]
    mlstm = case["type"] == "mlstm"
    n, dim, vdim = (memory_heads, 256, 512) if mlstm else (heads, 128, 128)
    out, states = [], []
    for x in torch.split(h, new):
        T = x.shape[0]
        q, k, v = ((x @ W[p + name].T).view(T, n, d) for name, d in (("q", dim), ("k", dim), ("v", vdim)))
        S = torch.zeros((n, vdim, dim), dtype=h.dtype, device=h.device)
        read = torch.zeros((T, n, vdim), dtype=h.dtype, device=h.device)
        if mlstm:
            q = q * dim ** -0.5
            log_in, log_forget = (15.0 * torch.tanh((x @ W[p + name].T + W[p + name + ".b"]) / 15.0) for name in ("i", "f"))
            log_forget = torch.nn.functional.logsigmoid(log_forget)
            norm, m = torch.zeros((n, dim), dtype=h.dtype, device=h.device), torch.zeros(n, dtype=h.dtype, device=h.device)
            for t in range(T):
                m_new = torch.maximum(log_forget[t] + m, log_in[t])
                keep, take = torch.exp(log_forget[t] + m - m_new), torch.exp(log_in[t] - m_new)
                S = keep[:, None, None] * S + v[t][:, :, None] * (take[:, None] * k[t])[:, None, :]
                norm, m = keep[:, None] * norm + take[:, None] * k[t], m_new
                read[t] = torch.einsum("hvd,hd->hv", S, q[t]) / (torch.maximum((norm * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
            normed = _rms(read, None, 1e-5).reshape(T, -1) * W[p + "norm"]
            states.append(torch.cat([S.reshape(n, -1), norm, m[:, None]], dim=1).reshape(-1))
        else:
            q, k, v = _silu(q), _silu(k), _silu(v)
            decay = torch.tensor(_decays(heads), dtype=h.dtype, device=h.device)
            for t in range(T):
                S = decay[:, None, None] * S + v[t][:, :, None] * k[t][:, None, :]
                read[t] = torch.einsum("hvd,hd->hv", S, q[t])
            normed = _rms(read.reshape(T, -1), W[p + "norm"], 1e-5)
            states.append(S.reshape(-1))
        out.append((normed * torch.sigmoid(x @ W[p + "g"].T)) @ W[p + "o"].T)
    return [torch.cat(out), torch.stack(states)]


def _delta(h, W, case, new):
    heads, key_heads, dim, vdim, taps = _delta_sizes(case)
    out, states, tails = [], [], []
    for x in torch.split(h, new):
        T = x.shape[0]
        raw = {name: x @ W["m." + name].T for name in ("q", "k", "v")}
        passed = {}
        for name, values in raw.items():
            padded = torch.cat([torch.zeros((taps - 1, values.shape[1]), dtype=h.dtype, device=h.device), values])
            passed[name] = _silu(sum(padded[i : i + T] * W[f"m.{name}.conv"][:, i] for i in range(taps)))
        tails.append(torch.cat([torch.cat([torch.zeros((taps - 1, raw[name].shape[1]), dtype=h.dtype, device=h.device), raw[name]])[-(taps - 1) :] for name in ("q", "k", "v")], dim=1))
        unit = [y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (passed["q"].view(T, key_heads, dim), passed["k"].view(T, key_heads, dim))]
        q, k = (y.repeat_interleave(heads // key_heads, dim=1) for y in (unit[0] * dim ** -0.5, unit[1]))
        v = passed["v"].view(T, heads, vdim)
        beta = torch.sigmoid(x @ W["m.b"].T)
        decay = torch.exp(-torch.exp(W["m.A_log"]) * torch.nn.functional.softplus(x @ W["m.a"].T + W["m.dt_bias"]))
        S = torch.zeros((heads, vdim, dim), dtype=h.dtype, device=h.device)
        read = torch.zeros((T, heads, vdim), dtype=h.dtype, device=h.device)
        for t in range(T):
            S = decay[t][:, None, None] * S
            update = beta[t][:, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + update[:, :, None] * k[t][:, None, :]
            read[t] = torch.einsum("hvd,hd->hv", S, q[t])
        features = (_rms(read, W["m.norm"], 1e-5) * _silu((x @ W["m.g"].T).view(T, heads, vdim))).reshape(T, -1)
        out.append(features @ W["m.o"].T)
        states.append(S.reshape(-1))
    return [torch.cat(out), torch.stack(states), torch.stack(tails)]


def _experts(h, W, p):
    scores = torch.sigmoid(h @ W[p + "router"].T)
    chosen = torch.topk(scores + W[p + "correction"], TOP, dim=-1).indices

    def expert(x, name):
        return (_silu(x @ W[p + name + ".gate"].T) * (x @ W[p + name + ".up"].T)) @ W[p + name + ".down"].T

    out = torch.sigmoid(h @ W[p + "shared.sg"].T) * expert(h, "shared")
    for e in range(EXPERTS):
        rows, _ = torch.nonzero(chosen == e, as_tuple=True)
        if rows.numel():
            out[rows] += scores[rows, e][:, None] * expert(h[rows], f"e{e}")
    return out


class _Wide:
    """The weights, widened to 64 bits one at a time as they are used."""

    def __init__(self, weights):
        self.weights = weights

    def __getitem__(self, name):
        return self.weights[name].double()


def exact(case, seed):
    generator = _generator(seed)
    raw = _weights(case, generator)
    W, kind = _Wide(raw), case["kind"]
    if kind in ("decode", "latent_decode"):
        contexts = _contexts(case)
        caches = []
        for _ in range(case["layers"]):
            if kind == "decode":
                shape = (QWEN3[case["shape"]][2], 128)
                caches.append([(_cached_rows(generator, c, *shape), _cached_rows(generator, c, *shape)) for c in contexts])
            else:
                caches.append([_cached_rows(generator, c, 576) for c in contexts])
        tokens = torch.randint(0, 32768, (case["batch"],), generator=generator, device="cuda")
        if kind == "decode":
            x = raw["model.embed_tokens.weight"][tokens].double()
            for i in range(case["layers"]):
                p = f"model.layers.{i}."
                h = _rms(x, W[p + "input_layernorm.weight"], 1e-6)
                x = x + torch.cat([_qwen3_attention(h[j : j + 1], W, p, case, caches[i][j][0].double(), caches[i][j][1].double(), c) for j, c in enumerate(contexts)])
                x = x + _qwen3_mlp(_rms(x, W[p + "post_attention_layernorm.weight"], 1e-6), W, p)
            head = "model.embed_tokens.weight" if QWEN3[case["shape"]][4] else "lm_head.weight"
            return _rms(x, W["model.norm.weight"], 1e-6) @ W[head].T
        x = raw["embed"][tokens].double()
        for i in range(case["layers"]):
            h = _rms(x, W[f"l{i}.norm1"], 1e-5)
            x = x + torch.cat([_latent(h[j : j + 1], W, f"l{i}.mix.", FASESUN[case["width"]][0], caches[i][j].double(), c)[0] for j, c in enumerate(contexts)])
        return _rms(x, W["final.norm"], 1e-5) @ W["embed"].T
    if kind == "experts":
        return _experts(_hidden(case, case["tokens"], case["width"], generator).double(), W, "l0.mlp.")
    new, cached = _lengths(case)
    if kind == "layer":
        width, _, kv_heads, _, _ = QWEN3[case["shape"]]
        pairs = [(_cached_rows(generator, c, kv_heads, 128).double(), _cached_rows(generator, c, kv_heads, 128).double()) for c in cached]
        second = _hidden(case, sum(new), width, generator).double()
        hidden = _hidden(case, sum(new), width, generator).double()
        attended = [_qwen3_attention(x, W, "model.layers.0.", case, *pair, c) for x, pair, c in zip(torch.split(hidden, new), pairs, cached)]
        return [torch.cat(attended), _qwen3_mlp(second, W, "model.layers.0."), None, None]      # the cache's pages are laid out by the library
    hidden = _hidden(case, sum(new), case["width"], generator).double()
    if kind == "latent":
        heads = FASESUN[case["width"]][0]
        empty = torch.zeros((0, 576), dtype=torch.float64, device="cuda")
        return [torch.cat([_latent(x, W, "l0.mix.", heads, empty, 0)[0] for x in torch.split(hidden, new)]), None]
    if kind == "memory":
        return _memory(hidden, W, "l0.mix.", case, new)
    return _delta(hidden, W, case, new)
