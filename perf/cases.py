"""The work that programs have this framework do, as cases that can be timed and compared.

A case is one layer of a served model (or a whole model) on one step's tokens: ``requests`` portions of about ``tokens`` new
tokens each, behind about ``context`` tokens that the request's cache holds already.  A step of single tokens behind a context is
decoding; a longer portion is (part of) a prompt; where there are several requests their lengths differ, as they do when prompts and
contexts of different users share a step.  Sizes are those of the random-weight presets (width 1024: the 350M shapes, 1536: the
700M shape, 2048: the 1.2B shapes).

The layers go through the parts (``build_part(...).forward``) with the cache manager's views and the batch builder's
description, as the framework's own step function calls them; the whole models through ``Engine.admit / step / release``.
"""

import math

import torch

DEVICE = "cuda"
VOCAB = 65536
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
PAGE = 16

# ------------------------------------------------------------------------------------------------------------------ cases


def _case(name, kind, width, requests, tokens, context, dtype="bfloat16"):
    return {"name": name, "kind": kind, "width": width, "requests": requests, "tokens": tokens, "context": context, "dtype": dtype}


def listed():
    return [
        # one user's next token through a feed-forward: the smallest call, two launches
        _case("mlp_decode_1", "gated_mlp", 1024, 1, 1, 0),
        # eight users decoding, each 4,096 tokens into a conversation: one attention layer
        _case("attention_decode_8x4096", "attention", 2048, 8, 1, 4096),
        # a prompt of ordinary length in one step: one attention layer
        _case("attention_prompt_2048", "attention", 2048, 1, 2048, 0),
        # an odd number of tokens of a few short prompts through the 700M shape's feed-forward
        _case("mlp_prompts_3x259", "gated_mlp", 1536, 3, 259, 0),
        # routed experts: eight users decoding, then a prompt
        _case("routed_decode_8", "routed_mlp", 2048, 8, 1, 0),
        _case("routed_prompt_2048", "routed_mlp", 2048, 1, 2048, 0),
        # the gated delta rule over a prompt
        _case("delta_prompt_2048", "gated_delta", 2048, 1, 2048, 0),
        # gated linear attention over two ragged prompts that go on from an earlier portion
        _case("gla_prompts_2x1501", "gated_linear", 1024, 2, 1501, 333),
        # latent attention: a later portion of a prompt behind what is cached
        _case("latent_portion_1023", "latent_attention", 2048, 1, 1023, 1500),
        # sigmoid attention with pooled blocks behind its window: a prompt longer than the window
        _case("pooled_prompt_3000", "pooled_attention", 2048, 1, 3000, 0),
        # the 32-bit path, which traces are compared on: a short prompt
        _case("attention_float32_300", "attention", 1024, 1, 300, 100, "float32"),
        # a whole small model serving eight short prompts together, then sixteen steps of decoding
        {**_case("serve_350m_8x96", "model", 1024, 8, 96, 0), "new_tokens": 16},
    ]


# how often a kind is drawn: about as often as the seven architectures' layers use it
_KINDS = (["attention"] * 4 + ["gated_mlp"] * 3 + ["short_conv"] * 2 + ["routed_mlp"] * 4 + ["gated_delta"] * 2 + ["retention"] * 2
          + ["gated_linear"] * 2 + ["latent_attention"] * 3 + ["pooled_attention"] * 2 + ["head"] + ["model"])


def draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(_KINDS)
    dtype = "float32" if rng.random() < 0.1 else "bfloat16"
    width = rng.choice([1024, 1536, 2048] if kind in ("attention", "short_conv", "gated_mlp", "head") else [1024, 2048])
    most = 256 if dtype == "float32" else 4096   # the 32-bit path is for short traces
    if kind == "model":
        return {"kind": kind, "width": 1024, "requests": spread(1, 16), "tokens": spread(1, 256), "context": 0, "dtype": "bfloat16", "new_tokens": spread(1, 24)}
    if rng.random() < 0.35:   # decoding
        requests, tokens, context = spread(1, 64), 1, spread(16, 4096 if dtype == "bfloat16" else 512)
        context = min(context, 65536 // requests)
    else:
        total = spread(2, most)
        requests = min(total, rng.choice([1, 1, 1, 2, 3, 5]))
        tokens, context = max(1, total // requests), rng.choice([0, 0, spread(1, 4096 if dtype == "bfloat16" else 512)])
    if kind in ("gated_mlp", "routed_mlp", "head"):
        context = 0
    if kind == "head":   # logits are wanted at a few places of a step
        requests, tokens = spread(1, 64), 1
    return {"kind": kind, "width": width, "requests": requests, "tokens": tokens, "context": context, "dtype": dtype}


def _ragged(length, requests):
    """``length`` for the first request, less for those after it, down to about half."""
    return [max(min(length, 1), length - length * i // (2 * requests)) for i in range(requests)]


def _portions(case):
    return _ragged(case["tokens"], case["requests"])


def _contexts(case):
    return _ragged(case["context"], case["requests"])


# ---------------------------------------------------------------------------------------------------- sizes of the layers
_FF = {1024: 4608, 1536: 6912, 2048: 8192}
EXPERTS, TOP, GROUPS, KEPT = 16, 4, 4, 2
HEADS8, VDIM, RANK, TAPS = 8, 128, 64, 4   # the recurrent mixers' heads, value channels, bottleneck, taps
LATENT = {"heads": 16, "dim": 64, "rope": 32, "vdim": 64, "rank": 256, "window": 2048, "theta": 10000.0}
POOLED = {"heads": 16, "groups": 4, "dim": 64, "window": 1024, "pool": 8, "cap": 30.0, "theta": 1000000.0}
LAYERS, ATTENTION_LAYERS = 16, (2, 5, 8, 10, 12, 14)
TAU = 16.0


def _key_dim(width):
    return 64 if width == 1024 else 128


def _decays():
    return tuple(1.0 - 2.0 ** (-5 - head) for head in range(HEADS8))


def _shapes(kind, width):
    """The tensors of a layer: local name -> (shape, role); ``m``: a matrix, ``1``: a vector near one, ``v``: a vector."""
    dk, heads = _key_dim(width), width // 64
    if kind == "gated_mlp":
        return {"gate_proj": ((_FF[width], width), "m"), "up_proj": ((_FF[width], width), "m"), "down_proj": ((width, _FF[width]), "m")}
    if kind == "attention":
        return {"q_proj": ((width, width), "m"), "k_proj": ((512, width), "m"), "v_proj": ((512, width), "m"), "out_proj": ((width, width), "m"),
                "q_norm": ((64,), "1"), "k_norm": ((64,), "1")}
    if kind == "short_conv":
        return {"in_proj": ((3 * width, width), "m"), "conv_weight": ((width, 3), "v"), "out_proj": ((width, width), "m")}
    if kind == "routed_mlp":
        ff = _FF[width] // TOP
        shapes = {"router": ((EXPERTS, width), "m")}
        for e in range(EXPERTS):
            shapes.update({f"experts.{e}.gate_proj": ((ff, width), "m"), f"experts.{e}.up_proj": ((ff, width), "m"), f"experts.{e}.down_proj": ((width, ff), "m")})
        return shapes
    if kind == "gated_delta":
        return {"q_proj": ((HEADS8 * dk, width), "m"), "k_proj": ((HEADS8 * dk, width), "m"), "v_proj": ((HEADS8 * VDIM, width), "m"),
                "q_conv": ((HEADS8 * dk, TAPS), "v"), "k_conv": ((HEADS8 * dk, TAPS), "v"), "v_conv": ((HEADS8 * VDIM, TAPS), "v"),
                "beta_proj": ((HEADS8, width), "m"), "a_log": ((HEADS8,), "v"), "dt_bias": ((HEADS8 * dk,), "v"),
                "decay_down": ((RANK, width), "m"), "decay_up": ((HEADS8 * dk, RANK), "m"), "gate_down": ((RANK, width), "m"),
                "gate_up": ((HEADS8 * VDIM, RANK), "m"), "out_norm": ((VDIM,), "1"), "out_proj": ((width, HEADS8 * VDIM), "m")}
    if kind in ("retention", "gated_linear"):
        shapes = {"q_proj": ((HEADS8 * dk, width), "m"), "k_proj": ((HEADS8 * dk, width), "m"), "v_proj": ((HEADS8 * VDIM, width), "m"),
                  "gate_proj": ((HEADS8 * VDIM, width), "m"), "out_proj": ((width, HEADS8 * VDIM), "m")}
        if kind == "gated_linear":
            shapes.update({"decay_down": ((RANK, width), "m"), "decay_up": ((HEADS8 * dk, RANK), "m"), "decay_bias": ((HEADS8 * dk,), "v"), "out_norm": ((VDIM,), "1")})
        return shapes
    if kind == "latent_attention":
        c = LATENT
        return {"q_proj": ((c["heads"] * (c["dim"] + c["rope"]), width), "m"), "down_proj": ((c["rank"] + c["rope"], width), "m"), "latent_norm": ((c["rank"],), "1"),
                "key_up_proj": ((c["heads"] * c["dim"], c["rank"]), "m"), "value_up_proj": ((c["heads"] * c["vdim"], c["rank"]), "m"),
                "gate_proj": ((c["heads"] * c["vdim"], width), "m"), "out_proj": ((width, c["heads"] * c["vdim"]), "m")}
    if kind == "pooled_attention":
        c = POOLED
        return {"q_proj": ((c["heads"] * c["dim"], width), "m"), "k_proj": ((c["groups"] * c["dim"], width), "m"), "v_proj": ((c["groups"] * c["dim"], width), "m"),
                "out_proj": ((width, c["heads"] * c["dim"]), "m"), "head_bias": ((c["heads"],), "v")}
    if kind == "head":
        return {"weight": ((VOCAB, width), "m")}
    raise ValueError(kind)


def _model_shapes(width):
    """The tensors of the whole model: (path, local name) -> (shape, role)."""
    shapes = {(("embedding",), "weight"): ((VOCAB, width), "e"), (("final_norm",), "scale"): ((width,), "1")}
    for i in range(LAYERS):
        for local, what in _shapes("attention" if i in ATTENTION_LAYERS else "short_conv", width).items():
            shapes[(("layers", i, "mixer"), local)] = what
        for local, what in _shapes("gated_mlp", width).items():
            shapes[(("layers", i, "ffn"), local)] = what
        shapes[(("layers", i, "pre_mixer_norm"), "scale")] = ((width,), "1")
        shapes[(("layers", i, "pre_ffn_norm"), "scale")] = ((width,), "1")
    return shapes


def _weights(shapes, dtype, generator):
    """Matrices of spread fan_in ** -0.5 in the compute type (in a whole model those that write to the residual stream divided by
    the square root of their number, as models of some depth are initialised), vectors in 32-bit."""
    tensors = {}
    for name, (shape, role) in shapes.items():
        values = torch.randn(shape, generator=generator, device=DEVICE)
        if role == "m":
            writes = isinstance(name, tuple) and name[1] in ("out_proj", "down_proj")
            tensors[name] = (values * (shape[1] * (2 * LAYERS if writes else 1)) ** -0.5).to(dtype)
        elif role == "e":
            tensors[name] = (values * 0.5).to(dtype)
        else:
            tensors[name] = 1 + 0.1 * values if role == "1" else 0.4 * values
    return tensors


def _inputs(case, seed):
    """The layer's tensors, and per request its rows (those behind which the step runs, then the step's)."""
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    tensors = _weights(_shapes(case["kind"], case["width"]), dtype, generator)
    rows = [torch.randn(c + n, case["width"], generator=generator, device=DEVICE).to(dtype) for c, n in zip(_contexts(case), _portions(case))]
    return tensors, rows


def _model_inputs(case, seed):
    generator = torch.Generator(device=DEVICE).manual_seed(seed)
    tensors = _weights(_model_shapes(case["width"]), DTYPES[case["dtype"]], generator)
    ids = [torch.randint(VOCAB, (n + case["new_tokens"],), generator=generator, device=DEVICE).tolist() for n in _portions(case)]
    return tensors, ids


# ---------------------------------------------------------------------------------------------------------------- prepare


def _spec(kind, width):
    from lalamo_b200.config import plan

    dk, heads = _key_dim(width), width // 64
    if kind == "gated_mlp":
        return plan.GatedMLPSpec(model_dim=width, hidden_dim=_FF[width])
    if kind == "attention":
        norm = plan.RMSNormSpec(dim=64, eps=1e-5)
        return plan.AttentionSpec(model_dim=width, num_heads=heads, num_groups=8, head_dim=64, qk_norm=norm, position=plan.RopeSpec(rotary_dim=64, theta=1000000.0))
    if kind == "short_conv":
        return plan.ShortConvSpec(model_dim=width, kernel_size=3)
    if kind == "routed_mlp":
        return plan.RoutedMLPSpec(model_dim=width, hidden_dim=_FF[width] // TOP, num_experts=EXPERTS, top=TOP, group_count=GROUPS, group_keep=KEPT)
    if kind == "gated_delta":
        return plan.GatedDeltaSpec(model_dim=width, num_heads=HEADS8, num_groups=HEADS8, key_dim=dk, value_dim=VDIM, conv_taps=TAPS, decay_rank=RANK, gate_rank=RANK)
    if kind == "retention":
        return plan.LinearAttentionSpec(model_dim=width, num_heads=HEADS8, key_dim=dk, value_dim=VDIM, decay="fixed", decay_values=_decays())
    if kind == "gated_linear":
        return plan.LinearAttentionSpec(model_dim=width, num_heads=HEADS8, key_dim=dk, value_dim=VDIM, decay="channel", decay_rank=RANK, tau=TAU, scaled="query", norm_weight=True)
    if kind == "latent_attention":
        c = LATENT
        return plan.LatentAttentionSpec(model_dim=width, num_heads=c["heads"], head_dim=c["dim"], rope_dim=c["rope"], value_dim=c["vdim"], latent_dim=c["rank"],
                                        latent_norm=plan.RMSNormSpec(dim=c["rank"], eps=1e-6, exact=True),
                                        position=plan.RopeSpec(rotary_dim=c["rope"], theta=c["theta"]), window=c["window"], gated=True)
    if kind == "pooled_attention":
        c = POOLED
        return plan.PooledWindowAttentionSpec(model_dim=width, num_heads=c["heads"], num_groups=c["groups"], head_dim=c["dim"], value_dim=c["dim"],
                                              position=plan.RopeSpec(rotary_dim=c["dim"], theta=c["theta"]), rotate_values=True, window=c["window"], pool=c["pool"],
                                              softcap=c["cap"], head_bias=True)
    return plan.HeadSpec(vocab_size=VOCAB, model_dim=width, tied=False)


def _plain(out):
    """A part may hand its output on as a sum that its consumer finishes."""
    return out if isinstance(out, torch.Tensor) else out.sum()


def _leaves(view):
    if view is None:
        return []
    if hasattr(view, "views"):
        return [tensor for one in view.views for tensor in _leaves(one)]
    return [getattr(view, name) for name in ("state", "k_pages", "v_pages") if getattr(view, name, None) is not None]


def prepare(case, seed):
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    from lalamo_b200 import ops
    from lalamo_b200.cache import CacheManager
    from lalamo_b200.engine import StepEntry
    from lalamo_b200.engine.executor import BatchBuilder
    from lalamo_b200.parts import Runtime, build_part

    ops.configure_matmul_precision()
    tensors, rows = _inputs(case, seed)
    runtime = Runtime(device=torch.device("cuda:0"), dtype=DTYPES[case["dtype"]])
    part = build_part(_spec(case["kind"], case["width"]), tensors, runtime)
    contexts, portions = _contexts(case), _portions(case)
    state = {"part": part, "runtime": runtime, "step": None, "view": None, "kept": []}
    state["x"] = torch.cat([row[c:] for row, c in zip(rows, contexts)])
    if not hasattr(part, "cache_need"):
        return state
    pages = sum(-(-(c + n) // PAGE) for c, n in zip(contexts, portions))
    cache = CacheManager([part.cache_need()], [None], runtime, page_size=PAGE, num_pages=pages, num_slots=case["requests"])
    builder = BatchBuilder(cache, runtime.device, VOCAB, planners=[part])
    slots = {}
    for i in range(case["requests"]):
        slots[cache.admit(i).slot] = i
    order = [slots[slot] for slot in range(case["requests"])]   # the request of number i has the state slot i

    def step(lengths):
        built = builder.build([StepEntry(order[i], [0] * n) for i, n in enumerate(lengths) if n])
        view = cache.views(built.block_tables, built.inputs.segment_slot)[0]
        return built.inputs, view

    if any(contexts):
        inputs, view = step(contexts)
        part.forward(torch.cat([row[:c] for row, c in zip(rows, contexts)]), inputs, view)
        for i, c in enumerate(contexts):
            cache.commit(order[i], c)
    state["step"], state["view"] = step(portions)
    state["kept"] = _leaves(state["view"])
    state["cache"] = cache
    return state


def _prepare_model(case, seed):
    from lalamo_b200.config.registry import config_from_dict
    from lalamo_b200.engine import Engine, EngineConfig
    from lalamo_b200.model_registry import PRESETS

    tensors, ids = _model_inputs(case, seed)
    config = config_from_dict(PRESETS["lfm2-350m"])
    held = sum(-(-len(one) // PAGE) * PAGE for one in ids)
    engine = Engine(config.to_plan(), tensors, EngineConfig(dtype=case["dtype"], page_size=PAGE, max_tokens=held, max_requests=case["requests"], freeze_gc=False), config)
    return {"engine": engine, "ids": ids, "prompts": _portions(case), "new_tokens": case["new_tokens"]}


# -------------------------------------------------------------------------------------------------------------------- run


def run(state):
    if "engine" in state:
        return _run_model(state)
    part = state["part"]
    if state["step"] is None:
        return [_plain(part.forward(state["x"]))]
    out = part.forward(state["x"], state["step"], state["view"])
    return [_plain(out)] + state["kept"]   # the layer's output, and the states or pages it has written


def _run_model(state):
    from lalamo_b200.engine import StepEntry

    engine, ids, prompts = state["engine"], state["ids"], state["prompts"]
    for i in range(len(ids)):
        engine.admit(i)
    logits = [engine.step([StepEntry(i, one[:n], [n - 1]) for i, (one, n) in enumerate(zip(ids, prompts))]).clone()]
    for k in range(state["new_tokens"]):
        logits.append(engine.step([StepEntry(i, [one[n + k]], [0]) for i, (one, n) in enumerate(zip(ids, prompts))]).clone())
    for i in range(len(ids)):
        engine.release(i)
    return logits


# ------------------------------------------------------------------------------------------------------------------- work


def work(case):
    kind, width, size = case["kind"], case["width"], DTYPES[case["dtype"]].itemsize
    contexts, portions = _contexts(case), _portions(case)
    tokens = sum(portions)
    numel = lambda shapes: sum(math.prod(shape) for shape, _ in shapes.values())  # noqa: E731
    seen = sum(n * c + n * (n + 1) // 2 for c, n in zip(contexts, portions))   # pairs of a token and one it sees
    if kind == "model":
        weights, steps = numel(_model_shapes(width)), 1 + case["new_tokens"]
        columns = weights - VOCAB * width
        every, wanted = tokens + case["requests"] * case["new_tokens"], case["requests"] * steps
        longest = [n + case["new_tokens"] for n in portions]
        pairs = sum(n * (n + 1) // 2 for n in longest)
        rows = sum(n + sum(range(n + 1, m + 1)) for n, m in zip(portions, longest))   # cached rows read: once a step
        return {"bytes": steps * weights * size + rows * len(ATTENTION_LAYERS) * 1024 * size + wanted * VOCAB * 4,
                "flops": 2 * columns * every + 2 * VOCAB * width * wanted + 4 * pairs * width * len(ATTENTION_LAYERS)}
    weights = numel(_shapes(kind, width))
    flops, moved = 2 * weights * tokens, weights * size + 2 * tokens * width * size
    dk = _key_dim(width)
    if kind == "routed_mlp":
        used = EXPERTS * (1 - (1 - TOP / EXPERTS) ** tokens)   # experts that some token chooses, on average
        per_expert = 3 * width * _FF[width] // TOP
        flops = 2 * tokens * (TOP * per_expert + EXPERTS * width)
        moved -= (EXPERTS - used) * per_expert * size
    elif kind == "head":
        moved += tokens * (4 * VOCAB - width * size)
    elif kind == "attention":
        flops += 4 * seen * width
        moved += (sum(contexts) + tokens) * 1024 * size
    elif kind == "short_conv":
        moved += case["requests"] * 2 * 2 * width * size
    elif kind in ("gated_delta", "retention", "gated_linear"):
        flops += tokens * HEADS8 * dk * VDIM * (8 if kind == "gated_delta" else 5)
        moved += case["requests"] * 2 * HEADS8 * dk * VDIM * 4
    elif kind == "latent_attention":
        c = LATENT
        visible = sum(min(p + 1, c["window"]) for q, n in zip(contexts, portions) for p in range(q, q + n))
        flops += 2 * visible * c["heads"] * (2 * c["rank"] + c["rope"])
        moved += (sum(min(q, c["window"]) for q in contexts) + tokens) * (c["rank"] + c["rope"]) * size
    elif kind == "pooled_attention":
        c = POOLED
        visible = sum(min(p + 1, c["window"]) + max(0, p - c["window"] + 1) // c["pool"] for q, n in zip(contexts, portions) for p in range(q, q + n))
        flops += 4 * visible * c["heads"] * c["dim"]
        moved += sum(min(q, c["window"]) + max(0, q - c["window"]) // c["pool"] + n for q, n in zip(contexts, portions)) * c["groups"] * 2 * c["dim"] * size
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """About four times the error against 64 bits: 1.5e-6 in 32-bit (and for logits, 32-bit sums of exact products), 0.004 to 0.006 of a layer
    in bfloat16 and of a whole model."""
    if case["dtype"] == "float32" or case["kind"] == "head":
        return {"rel": 1e-5}
    return {"rel": 2e-2}


# ------------------------------------------------------------------------------------------------------ the same in 64 bits


def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _turn(x, positions, theta, sign=1.0):
    """Channel i of the last dimension with channel i + half, by position * theta ** (-2i / channels)."""
    channels = x.shape[-1]
    inverse = 1.0 / (torch.tensor(theta, dtype=torch.float64, device=x.device) ** (torch.arange(0, channels, 2, device=x.device, dtype=torch.float64) / channels))
    angle = (positions.double()[:, None] * inverse)[:, None, :]
    cos, sin = torch.cos(angle), sign * torch.sin(angle)
    u, v = x[..., : channels // 2], x[..., channels // 2 :]
    return torch.cat([u * cos - v * sin, v * cos + u * sin], dim=-1)


def _silu(z):
    return z * torch.sigmoid(z)


def _mlp(x, w):
    return (_silu(x @ w["gate_proj"].T) * (x @ w["up_proj"].T)) @ w["down_proj"].T


def _attention(x, w, first):
    """All positions' keys, the outputs from position ``first`` on."""
    n, width = x.shape
    heads, positions = width // 64, torch.arange(n, device=x.device)
    q = _turn(_rms((x[first:] @ w["q_proj"].T).view(-1, heads, 64), w["q_norm"], 1e-5), positions[first:], 1000000.0)
    k = _turn(_rms((x @ w["k_proj"].T).view(n, 8, 64), w["k_norm"], 1e-5), positions, 1000000.0)
    v = (x @ w["v_proj"].T).view(n, 8, 64)
    hidden = positions[None, :] > positions[first:, None]
    out = torch.empty_like(q)
    for h in range(heads):
        g = h // (heads // 8)
        out[:, h] = torch.softmax((q[:, h] @ k[:, g].T / 8).masked_fill(hidden, -math.inf), -1) @ v[:, g]
    return out.flatten(1) @ w["out_proj"].T


def _conv(x, taps):
    """Causal, depthwise: the last column of ``taps`` multiplies the row itself."""
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    return sum(padded[j : j + x.shape[0]] * taps[:, j] for j in range(n))


def _short_conv(x, w):
    b, c, u = (x @ w["in_proj"].T).chunk(3, dim=-1)
    u = b * u
    return (c * _conv(u, w["conv_weight"])) @ w["out_proj"].T, u[-2:]


def _routed(x, w):
    scores = torch.sigmoid(x @ w["router"].T)
    per_group = scores.view(-1, GROUPS, EXPERTS // GROUPS)
    kept = per_group.topk(2, dim=-1).values.sum(-1).topk(KEPT, dim=-1).indices
    open_ = torch.zeros(x.shape[0], GROUPS, dtype=torch.bool, device=x.device).scatter_(1, kept, True).repeat_interleave(EXPERTS // GROUPS, dim=1)
    weights, chosen = scores.masked_fill(~open_, -1.0).topk(TOP, dim=-1)
    out = torch.zeros_like(x)
    for e in range(EXPERTS):
        token, place = (chosen == e).nonzero(as_tuple=True)
        one = {name: w[f"experts.{e}.{name}"] for name in ("gate_proj", "up_proj", "down_proj")}
        out.index_add_(0, token, weights[token, place, None] * _mlp(x[token], one))
    return out


def _recurrence(q, k, v, decay, beta, first):
    """Read-outs from ``first`` on and the last state; ``beta``: the delta rule's correction (None: none)."""
    n, heads, dk = k.shape
    S, outs = q.new_zeros(heads, dk, v.shape[-1]), []
    for t in range(n):
        S = S * decay[t, :, :, None]
        u = v[t] if beta is None else beta[t, :, None] * (v[t] - (k[t, :, None, :] @ S)[:, 0])
        S = torch.baddbmm(S, k[t, :, :, None], u[:, None, :])
        if t >= first:
            outs.append((q[t, :, None, :] @ S)[:, 0])
    return torch.stack(outs), S


def _delta(x, w, first):
    n, dk = x.shape[0], w["q_proj"].shape[0] // HEADS8
    projected = torch.cat([x @ w[f"{one}_proj"].T for one in "qkv"], dim=-1)
    q, k, v = (_silu(_conv(x @ w[f"{one}_proj"].T, w[f"{one}_conv"])).view(n, HEADS8, -1) for one in "qkv")
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    rate = torch.exp(w["a_log"])[None, :, None]
    z = ((x @ w["decay_down"].T) @ w["decay_up"].T + w["dt_bias"]).view(n, HEADS8, dk)
    decay = torch.exp(-rate * torch.nn.functional.softplus(z, threshold=40.0))
    out, S = _recurrence(q, k, v, decay, torch.sigmoid(x @ w["beta_proj"].T), first)
    gate = torch.sigmoid((x[first:] @ w["gate_down"].T) @ w["gate_up"].T)
    return (_rms(out, w["out_norm"], 1e-6).flatten(1) * gate) @ w["out_proj"].T, S, projected


def _linear(x, w, first):
    n, dk = x.shape[0], w["q_proj"].shape[0] // HEADS8
    q, k, v = ((x @ w[f"{one}_proj"].T).view(n, HEADS8, -1) for one in "qkv")
    if "decay_up" in w:   # one decay per key channel, made from the token
        z = (x @ w["decay_down"].T) @ w["decay_up"].T + w["decay_bias"]
        decay, norm = (torch.sigmoid(z) ** (1.0 / TAU)).view(n, HEADS8, dk), w["out_norm"]
    else:
        decay, norm = torch.tensor(_decays(), dtype=x.dtype, device=x.device)[None, :, None].expand(n, HEADS8, dk), 1.0
    out, S = _recurrence(q * dk ** -0.5, k, v, decay, None, first)
    gated = _rms(out, norm, 1e-5).flatten(1) * _silu(x[first:] @ w["gate_proj"].T)
    if "decay_up" not in w:
        S = S * dk ** -0.5   # the scale is on the keys there
    return gated @ w["out_proj"].T, S


def _latent(x, w, first):
    c, n = LATENT, x.shape[0]
    heads, positions = c["heads"], torch.arange(n, device=x.device)
    q = (x[first:] @ w["q_proj"].T).view(-1, heads, c["dim"] + c["rope"])
    q_turned = _turn(q[..., c["dim"] :], positions[first:], c["theta"])
    down = x @ w["down_proj"].T
    latent = _rms(down[:, : c["rank"]], w["latent_norm"], 1e-6)
    turned = _turn(down[:, None, c["rank"] :], positions, c["theta"])[:, 0]
    keys = (latent @ w["key_up_proj"].T).view(n, heads, c["dim"])
    values = (latent @ w["value_up_proj"].T).view(n, heads, c["vdim"])
    distance = positions[first:, None] - positions[None, :]
    hidden = (distance < 0) | (distance >= c["window"])
    out = torch.empty(n - first, heads, c["vdim"], dtype=x.dtype, device=x.device)
    for h in range(heads):
        scores = (q[:, h, : c["dim"]] @ keys[:, h].T + q_turned[:, h] @ turned.T) * (c["dim"] + c["rope"]) ** -0.5
        out[:, h] = torch.softmax(scores.masked_fill(hidden, -math.inf), -1) @ values[:, h]
    return (out.flatten(1) * torch.sigmoid(x[first:] @ w["gate_proj"].T)) @ w["out_proj"].T


def _pooled(x, w, first):
    c, n = POOLED, x.shape[0]
    heads, groups, dim, positions = c["heads"], c["groups"], c["dim"], torch.arange(n, device=x.device)
    q = _turn((x[first:] @ w["q_proj"].T).view(-1, heads, dim), positions[first:], c["theta"])
    k = _turn((x @ w["k_proj"].T).view(n, groups, dim), positions, c["theta"])
    v = _turn((x @ w["v_proj"].T).view(n, groups, dim), positions, c["theta"])
    blocks = n // c["pool"]
    mean = lambda rows: rows[: blocks * c["pool"]].view(blocks, c["pool"], groups, dim).mean(1)  # noqa: E731
    keys, values = torch.cat([mean(k), k]), torch.cat([mean(v), v])
    distance = positions[first:, None] - positions[None, :]
    last = (torch.arange(blocks, device=x.device) + 1) * c["pool"] - 1
    seen = torch.cat([last[None, :] <= positions[first:, None] - c["window"], (distance >= 0) & (distance < c["window"])], dim=1)
    out = torch.empty_like(q)
    for h in range(heads):
        g = h // (heads // groups)
        scores = c["cap"] * torch.tanh(q[:, h] @ keys[:, g].T * dim ** -0.5 / c["cap"])
        out[:, h] = (torch.sigmoid(scores + w["head_bias"][h]) * seen) @ values[:, g]
    return _turn(out, positions[first:], c["theta"], -1.0).flatten(1) @ w["out_proj"].T


def _model(ids, w, wanted):
    x = w[(("embedding",), "weight")][torch.tensor(ids, device=DEVICE)]
    for i in range(LAYERS):
        own = lambda role: {local: tensor for (path, local), tensor in w.items() if path == ("layers", i, role)}  # noqa: E731, B023
        h = _rms(x, own("pre_mixer_norm")["scale"], 1e-5)
        x = x + (_attention(h, own("mixer"), 0) if i in ATTENTION_LAYERS else _short_conv(h, own("mixer"))[0])
        x = x + _mlp(_rms(x, own("pre_ffn_norm")["scale"], 1e-5), own("ffn"))
    return _rms(x[wanted:], w[(("final_norm",), "scale")], 1e-5) @ w[(("embedding",), "weight")].T


def exact(case, seed):
    kind = case["kind"]
    if kind == "model":
        tensors, ids = _model_inputs(case, seed)
        w = {name: tensor.double() for name, tensor in tensors.items()}
        rows = [_model(one, w, n - 1) for one, n in zip(ids, _portions(case))]
        return [torch.stack([row[k] for row in rows]) for k in range(1 + case["new_tokens"])]
    tensors, rows = _inputs(case, seed)
    w = {name: tensor.double() for name, tensor in tensors.items()}
    if kind in ("gated_mlp", "routed_mlp", "head"):
        x = torch.cat(rows).double()
        return [_mlp(x, w) if kind == "gated_mlp" else _routed(x, w) if kind == "routed_mlp" else x @ w["weight"].T]
    outs, states, inputs = [], [], []
    for row, first in zip(rows, _contexts(case)):
        x = row.double()
        if kind == "short_conv":
            out, last = _short_conv(x, w)
            outs.append(out[first:])
            states.append(torch.cat([last.new_zeros(max(0, 2 - len(last)), last.shape[1]), last]))
        elif kind == "gated_delta":
            out, S, projected = _delta(x, w, first)
            outs.append(out)
            states.append(S)
            last = projected[-(TAPS - 1) :]
            inputs.append(torch.cat([last.new_zeros(max(0, TAPS - 1 - len(last)), last.shape[1]), last]))
        elif kind in ("retention", "gated_linear"):
            out, S = _linear(x, w, first)
            outs.append(out)
            states.append(S)
        else:
            outs.append({"attention": _attention, "latent_attention": _latent, "pooled_attention": _pooled}[kind](x, w, first))
    found = [torch.cat(outs)]
    if states:
        found.append(torch.stack(states))
    elif kind == "latent_attention":
        found.append(None)
    else:
        found += [None, None]
    if inputs:
        found.append(torch.stack(inputs))
    return found
