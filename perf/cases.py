"""Speed cases: what a program that uses this framework has it do, from one decoded token to prompts of thousands.

Two kinds of case.  ``step``: a whole call of ``Engine.step`` (prompts, or one token for each of a batch of sequences that
already hold a context) on a model of one of the benchmark shapes; the answer is its logits.  ``layer``: one layer of one of the
designs, put together from the registered parts the way an arrangement does it (norm, mixer or feed-forward, and the norm
that takes its output into the stream); the answer is the stream, the normed rows and the states the layer carries on.

Every size is one of the benchmark shapes' (``thintensor_b200/config/shapes.json``) or a smaller model's of the same make.
"""
import math

import torch

from thintensor_b200.cache.cache import SequenceCache
from thintensor_b200.config.registry import load_config
from thintensor_b200.engine.context import StepContext, Workspace
from thintensor_b200.engine.engine import Entry
from thintensor_b200.engine.model import DecoderModel
from thintensor_b200.parts import FEED_FORWARDS, MIXERS, NORMS
from thintensor_b200.parts.base import Delta
from thintensor_b200.parts.spec import PartSpec
from thintensor_b200.runtime import Runtime

DEVICE = "cuda"
EPS = 1e-6
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
BLOCK = 64


# ---------------------------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # One user's chat, a token at a time: the smallest call there is, and the one whose latency is felt.
        {"name": "llama_decode_1", "kind": "step", "model": "llama", "layers": 16, "dtype": "bf16", "batch": 1, "context": 2048, "new": 1},
        # A server's decode step with many sequences: weights and cache weigh about the same.
        {"name": "llama_decode_64", "kind": "step", "model": "llama", "layers": 16, "dtype": "bf16", "batch": 64, "context": 2048, "new": 1},
        # A prompt of the headline benchmark's length through the whole model.
        {"name": "llama_prompt_2048", "kind": "step", "model": "llama", "layers": 16, "dtype": "bf16", "batch": 1, "context": 0, "new": 2048},
        # The exact 32-bit path, which is run to check other implementations: a short prompt of an odd length.
        {"name": "llama_fp32_prompt_193", "kind": "step", "model": "llama", "layers": 2, "dtype": "fp32", "batch": 1, "context": 0, "new": 193},
        # A decode step of the design whose layers are recurrences, attention beside one, and dense feed-forwards.
        {"name": "famalorn_decode_8", "kind": "step", "model": "famalorn", "layers": 6, "dtype": "bf16", "batch": 8, "context": 2000, "new": 1},
        # The same model's prompts: four of unequal lengths in one step.
        {"name": "famalorn_prompt_ragged", "kind": "step", "model": "famalorn", "layers": 3, "dtype": "bf16", "batch": 4, "context": 0, "new": 731},
        # Single layers on a prompt, one for each way to mix tokens that the designs have.
        {"name": "mamba2_prompt_2048", "kind": "layer", "part": "mamba2", "hidden": 2048, "heads": 64, "batch": 1, "new": 2048},
        {"name": "delta_prompt_4097", "kind": "layer", "part": "delta", "hidden": 2048, "heads": 16, "batch": 1, "new": 4097},
        {"name": "retention_prompt_4x1024", "kind": "layer", "part": "retention", "hidden": 2048, "heads": 16, "batch": 4, "new": 1024},
        {"name": "differential_prompt_2048", "kind": "layer", "part": "differential", "hidden": 2048, "heads": 16, "batch": 1, "new": 2048},
        # Routed experts: every design but the first keeps its feed-forwards in them.
        {"name": "moe_prompt_2048", "kind": "layer", "part": "moe", "hidden": 2048, "heads": 16, "batch": 1, "new": 2048},
        # Attention over cached latents, a decode step of a busy server.
        {"name": "latent_decode_48", "kind": "layer", "part": "latent", "hidden": 2048, "heads": 16, "batch": 48, "new": 1, "context": 1500},
    ]


def _spread(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    if rng.random() < 0.35:
        model = rng.choice(("llama", "llama", "famalorn"))
        dtype = "fp32" if rng.random() < 0.2 else "bf16"
        layers = 2 if dtype == "fp32" else rng.choice((3, 6))
        if rng.random() < 0.5:
            return {"kind": "step", "model": model, "layers": layers, "dtype": dtype, "batch": _spread(rng, 1, 8 if dtype == "fp32" else 64),
                    "context": _spread(rng, 60, 2100), "new": 1}
        return {"kind": "step", "model": model, "layers": layers, "dtype": dtype, "batch": rng.randint(1, 4), "context": 0,
                "new": _spread(rng, 2, 100 if dtype == "fp32" else 1000)}
    part = rng.choice(("mamba2", "delta", "retention", "lightning", "differential", "moe", "latent"))
    hidden = rng.choice((1024, 2048, 3072))
    heads = (hidden // 32 if rng.random() < 0.5 else hidden // 64) if part == "mamba2" else hidden // 128
    if part == "latent":
        return {"kind": "layer", "part": part, "hidden": hidden, "heads": heads, "batch": _spread(rng, 1, 64), "new": 1, "context": _spread(rng, 70, 3000)}
    batch = rng.choice((1, 1, 2, 3, 5))
    return {"kind": "layer", "part": part, "hidden": hidden, "heads": heads, "batch": batch, "new": _spread(rng, 9, 4200 // batch)}


def lengths(case):
    """How many tokens each sequence brings: prompts that share a step are rarely of one length."""
    new, batch = case["new"], case["batch"]
    if new == 1 or case["kind"] == "layer":
        return [new] * batch
    return [max(1, new - 97 * i if i % 2 else new + 61 * i) for i in range(batch)]


# ------------------------------------------------------------------------------------------------- weights and inputs

LLAMA = {"architectures": ["LlamaForCausalLM"], "model_type": "llama", "vocab_size": 128256, "rope_theta": 500000.0, "rms_norm_eps": 1e-5,
         "max_position_embeddings": 131072, "num_key_value_heads": 8, "hidden_size": 2048, "num_attention_heads": 32, "head_dim": 64,
         "intermediate_size": 8192, "tie_word_embeddings": True,
         "rope_scaling": {"rope_type": "llama3", "factor": 32.0, "low_freq_factor": 1.0, "high_freq_factor": 4.0,
                          "original_max_position_embeddings": 8192}}
FAMALORN = [
    {"type": "delta", "mlp": {"kind": "dense", "ff": 8192}, "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}},
    {"type": "mamba2", "mlp": {"kind": "dense", "ff": 8192}, "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4}},
    {"type": "parallel", "mlp": {"kind": "dense", "ff": 8192}, "mixer": {
        "left": {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 64, "scale": 0.125, "rot": {"dims": 32, "base": 500000.0}},
        "right": {"heads": 32, "vdim": 64, "state": 64, "groups": 1, "norm_groups": 1, "conv": 4}, "left_scale": 1.0, "right_scale": 1.0}},
]


def _config(case):
    if case["model"] == "llama":
        return {**LLAMA, "num_hidden_layers": case["layers"]}
    return {"architecture": "Famalorn", "vocab": 128256, "width": 2048, "norm": {"eps": EPS}, "layers": [FAMALORN[i % 3] for i in range(case["layers"])]}


def _decays(heads):
    return [1.0 - 2.0 ** (-5.0 - 3.0 * i / max(1, heads - 1)) for i in range(heads)]


def _part(case):
    """Role, kind and sizes of a layer's part, as the designs' descriptions have them."""
    hidden, heads = case["hidden"], case["heads"]
    if case["part"] == "mamba2":
        return MIXERS, "mamba2", {"hidden": hidden, "heads": heads, "head_dim": 64, "state": 128, "groups": 1, "norm_groups": 1, "conv": 4, "eps": EPS}
    if case["part"] == "delta":
        return MIXERS, "gated_delta", {"hidden": hidden, "heads": heads, "qk_heads": heads // 2, "key_dim": 128, "value_dim": 128, "conv": 4, "eps": EPS}
    if case["part"] == "lightning":
        return MIXERS, "decay_linear_attention", {"hidden": hidden, "heads": heads, "key_dim": 128, "value_dim": 128, "decay": _decays(heads),
                                                  "activation": "silu", "norm": "all", "norm_weight": True, "gate": "sigmoid", "eps": EPS}
    if case["part"] == "retention":
        position = PartSpec("rope", {"head_dim": 128, "theta": 10000.0, "rotary_dim": 128, "table_precision": "float64"})
        return MIXERS, "decay_linear_attention", {"hidden": hidden, "heads": heads, "key_dim": 128, "value_dim": 256, "decay": _decays(heads),
                                                  "position": position, "key_scale": 128 ** -0.5, "norm": "head", "gate": "silu", "eps": EPS}
    if case["part"] == "differential":
        return MIXERS, "differential_attention", {"hidden": hidden, "heads": heads, "kv_heads": heads // 4, "dim": 64, "value_dim": 128, "scale": 0.125,
                                                  "diff": 0.2, "eps": 1e-5, "bias": True, "q_gain": (0.1, 1024)}
    if case["part"] == "latent":
        position = PartSpec("rope", {"head_dim": 64, "theta": 10000.0, "rotary_dim": 64, "table_precision": "float64"})
        return MIXERS, "latent_attention", {"hidden": hidden, "heads": heads, "dim": 64, "rot_dim": 64, "value_dim": 128, "q_rank": hidden * 3 // 8,
                                            "kv_rank": 512, "scale": 128 ** -0.5, "eps": EPS, "position": position, "window": 1024}
    if case["part"] == "moe":
        return FEED_FORWARDS, "moe", {"hidden": hidden, "experts": 16, "top": 4, "inter": 1024, "groups": 4, "keep": 2, "shared_inter": 2 * hidden}
    raise KeyError(case["part"])


def _tensor(name, decl, generator, dtype):
    """A checkpoint's tensor: matrices N(0, 0.02), norm weights about one, decays and step sizes as such models are started with."""
    def uniform(a, b):
        return torch.rand(decl.shape, generator=generator, device=DEVICE) * (b - a) + a

    last = name.rsplit(".", 1)[-1]
    if last == "A_log":
        value = uniform(1.0, 16.0).log()
    elif last == "dt_bias":                                     # softplus of it lies between 0.001 and 0.1
        value = uniform(math.log(0.001), math.log(0.1)).exp()
        value = value + torch.log(-torch.expm1(-value))
    elif "conv" in name and len(decl.shape) == 2:
        value = 0.3 * torch.randn(decl.shape, generator=generator, device=DEVICE)
    elif decl.init == "norm":
        value = 1.0 + 0.1 * torch.randn(decl.shape, generator=generator, device=DEVICE)
    elif decl.init == "small" or len(decl.shape) == 1:
        value = 0.1 * torch.randn(decl.shape, generator=generator, device=DEVICE)
    else:
        value = 0.02 * torch.randn(decl.shape, generator=generator, device=DEVICE)
    return value.to(dtype)


def _tensors(decls, seed, dtype):
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(seed)
    return {name: _tensor(name, decl, generator, dtype) for name, decl in decls.items() if not decl.prefer_alias}


def _model(case):
    arch, config = load_config(_config(case))
    return arch, config, DecoderModel(arch.describe(config), DTYPES[case["dtype"]], DEVICE)


def _past(need, tokens, generator, dtype):
    """What earlier steps left in the cache for one sequence: keys and values."""
    k = torch.randn((need.kv_heads, tokens, need.head_dim), generator=generator, device=DEVICE).to(dtype)
    v = torch.randn((need.kv_heads, tokens, need.v_dim), generator=generator, device=DEVICE).to(dtype) if need.v_dim else None
    return k, v


def _state(need, batch, generator):
    return 0.5 * torch.randn((batch, *need.shape), generator=generator, device=DEVICE)


def _fill(cache, entry, slots, past, states):
    """Put contexts into the cache where steps would have left them."""
    view = cache.run_cache(entry)
    for i, (k, v) in enumerate(past or []):
        rows = cache.kv_groups[view.group].table.row(slots[i])
        begin = sum(1 for r in rows if r < 0)                  # blocks that a window has given back
        for number in range(begin, -(-k.shape[1] // BLOCK)):
            piece = slice(number * BLOCK, min((number + 1) * BLOCK, k.shape[1]))
            count = piece.stop - piece.start
            view.k_pool[rows[number], :, :count] = k[:, piece]
            if v is not None:
                view.v_pool[rows[number], :, :, :count] = v[:, piece].transpose(1, 2)
    for own, value in zip(cache.run_state(entry), states):
        own[slots] = value


def _step_inputs(case, model, seed):
    """Tokens, and what the sequences hold already: one entry for each run's mixers."""
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(seed * 7919 + 13)
    tokens = [torch.randint(0, 128256, (n,), generator=generator, device=DEVICE).tolist() for n in lengths(case)]
    kv, state, _ = model.cache_needs()
    past, states = [], []
    for entry in range(len(kv)):
        past.append([_past(kv[entry], case["context"], generator, DTYPES[case["dtype"]]) for _ in range(case["batch"])]
                    if kv[entry] is not None and case["context"] else None)
        states.append([_state(need, case["batch"], generator) if case["context"] else torch.zeros((case["batch"], *need.shape), device=DEVICE)
                       for need in state[entry]])
    return tokens, past, states


# ------------------------------------------------------------------------------------------------------------ prepare

def prepare(case, seed):
    return _prepare_step(case, seed) if case["kind"] == "step" else _prepare_layer(case, seed)


def _prepare_step(case, seed):
    arch, config, model = _model(case)
    model.bind(_tensors(model.weight_declarations(), seed, DTYPES[case["dtype"]]))
    batch, context = case["batch"], case["context"]
    most = max(lengths(case)) + context + BLOCK
    engine = Runtime(None, arch, config, model).new_engine(batch * (-(-most // BLOCK) * BLOCK), batch)
    tokens, past, states = _step_inputs(case, model, seed)
    slots = []
    if context:
        for _ in range(batch):
            slot = engine.open()
            engine.cache.reserve(slot, context + 1)
            engine.cache.lengths[slot] = context
            slots.append(slot)
        for entry in range(len(states)):
            _fill(engine.cache, entry, slots, past[entry], states[entry])
    return {"kind": "step", "engine": engine, "slots": slots, "tokens": tokens, "context": context}


def _prepare_layer(case, seed):
    registry, kind, sizes = _part(case)
    part = registry.build(kind, sizes)
    dtype, hidden, batch, new, context = torch.bfloat16, case["hidden"], case["batch"], case["new"], case.get("context", 0)
    weights = _tensors(part.weights(), seed, dtype)
    part.bind(weights, dtype, torch.device(DEVICE))
    before, after = NORMS.build("rmsnorm", {"dim": hidden, "eps": EPS}), NORMS.build("rmsnorm", {"dim": hidden, "eps": EPS})
    stream, norms, past, states = _layer_inputs(case, part, seed)
    before.bind({"weight": norms[0]}, dtype, DEVICE)
    after.bind({"weight": norms[1]}, dtype, DEVICE)
    cache = None
    tables = []
    slots = list(range(batch))
    if registry is MIXERS:
        need = part.cache_need()
        blocks = batch * -(-(context + new) // BLOCK)
        cache = SequenceCache([need], [part.state_needs()], [None], blocks, batch, dtype, DEVICE)
        slots = [cache.alloc_slot() for _ in range(batch)]
        for slot in slots:
            cache.reserve(slot, context + new)
            cache.lengths[slot] = context
        if context:
            _fill(cache, 0, slots, past, [])
        if need is not None:
            tables = [torch.tensor(cache.table_rows(0, slots, cache.max_blocks(slots)), dtype=torch.int32, device=DEVICE)]
    tokens = batch * new
    ints = lambda values: torch.tensor(values, dtype=torch.int32, device=DEVICE)
    ctx = StepContext(n_tokens=tokens, sequences=batch, decode=new == 1, max_new=new, max_total=context + new, tokens=torch.zeros(tokens, dtype=torch.int32, device=DEVICE),
                      cu=ints([i * new for i in range(batch + 1)]), len_before=ints([context] * batch), slots=ints(slots), tables=tables, act_dtype=dtype,
                      workspace=Workspace(torch.device(DEVICE)), status=torch.zeros(1, dtype=torch.int32, device=DEVICE))
    return {"kind": "layer", "part": part, "mixer": registry is MIXERS, "before": before, "after": after, "stream": stream, "cache": cache, "ctx": ctx,
            "residual": torch.empty_like(stream), "normed": torch.empty(stream.shape, dtype=dtype, device=DEVICE),
            "out": torch.empty(stream.shape, dtype=dtype, device=DEVICE)}


def _layer_inputs(case, part, seed):
    generator = torch.Generator(device=DEVICE)
    generator.manual_seed(seed * 7919 + 29)
    tokens, hidden = case["batch"] * case["new"], case["hidden"]
    stream = 0.02 * torch.randn((tokens, hidden), generator=generator, device=DEVICE)        # as an embedding of random weights leaves it
    norms = [1.0 + 0.1 * torch.randn(hidden, generator=generator, device=DEVICE) for _ in range(2)]
    past = None
    if case.get("context"):
        past = [_past(part.cache_need(), case["context"], generator, torch.bfloat16) for _ in range(case["batch"])]
    return stream, norms, past, []


# ---------------------------------------------------------------------------------------------------------------- run

def run(state):
    if state["kind"] == "step":
        engine = state["engine"]
        if state["context"]:
            # one more token for every sequence; the next pass continues from the same context
            logits = engine.step([Entry(slot, tokens, [0]) for slot, tokens in zip(state["slots"], state["tokens"])])
            for slot in state["slots"]:
                engine.cache.lengths[slot] = state["context"]
            return logits
        slots = [engine.open() for _ in state["tokens"]]
        logits = engine.step([Entry(slot, tokens, _wanted(len(tokens))) for slot, tokens in zip(slots, state["tokens"])])
        for slot in slots:
            engine.close(slot)
        return logits
    ctx, cache, residual = state["ctx"], state["cache"], state["residual"]
    residual.copy_(state["stream"])
    ctx.residual = residual                     # nothing else reads the stream before the next norm: the part may add into it
    ctx.memo.clear()
    state["before"].forward(ctx, residual, None, state["normed"])
    states = []
    if state["mixer"]:
        states = cache.run_state(0)
        for tensor in states:                   # the sequences are new
            tensor.zero_()
        delta = state["part"].forward(ctx, state["normed"], cache.run_cache(0), states)
    else:
        delta = state["part"].forward(ctx, state["normed"])
    state["after"].forward(ctx, residual, delta or Delta(None), state["out"])
    return {"stream": residual, "normed": state["out"], "states": list(states)}


def _wanted(n):
    """A prompt's logits: the last place, and places before it as a program that scores a text wants them."""
    return sorted({n - 1, n // 2, n // 3, 0})


# -------------------------------------------------------------------------------------------------------------- work

def work(case):
    if case["kind"] == "step":
        return _step_work(case)
    hidden, heads, batch, new, context = case["hidden"], case["heads"], case["batch"], case["new"], case.get("context", 0)
    tokens = batch * new
    bytes_, flops = tokens * hidden * (4 + 4 + 2), 0.0           # the stream in and out, the normed rows out
    part = case["part"]

    def matrix(rows, cols, share=1.0):
        nonlocal bytes_, flops
        bytes_ += 2 * rows * cols
        flops += 2.0 * tokens * rows * cols * share

    def states(count):                                          # a state's update and its reading: two multiply-adds a number
        nonlocal bytes_, flops
        bytes_ += 4 * batch * count
        flops += 4.0 * tokens * count

    if part == "mamba2":
        inner = heads * 64
        matrix(2 * inner + 256 + heads, hidden)
        states(heads * 64 * 128)
        matrix(hidden, inner)
    elif part == "delta":
        inner = heads * 128
        matrix(3 * inner + 2 * heads, hidden)
        states(heads * 128 * 128)
        flops += 2.0 * tokens * heads * 128 * 128               # and the state read by the key
        matrix(hidden, inner)
    elif part in ("lightning", "retention"):
        values = heads * (128 if part == "lightning" else 256)
        matrix(2 * heads * 128 + 2 * values, hidden)
        states(128 * values)
        matrix(hidden, values)
    elif part == "differential":
        matrix(heads * 128 + 2 * (heads // 4) * 128, hidden)
        matrix(hidden, heads * 128)
        flops += 2.0 * batch * new * (new + 1) / 2 * heads * (128 + 256)
        bytes_ += tokens * 2 * (heads // 4) * 128 * 2
    elif part == "latent":
        rank = hidden * 3 // 8
        matrix(rank + 576, hidden)
        matrix(heads * 128, rank)
        matrix(heads * 64 + heads * 128, 512)
        matrix(hidden, heads * 128)
        seen = min(1024, context + 1)
        bytes_ += batch * seen * 576 * 2
        flops += 2.0 * batch * seen * heads * (576 + 512)
    elif part == "moe":
        matrix(16, hidden)
        share = 1.0 - (0.75 ** tokens)                          # experts that some token chose
        bytes_ += 2 * 3 * hidden * (share * 16 * 1024 + 2 * hidden)
        flops += 2.0 * tokens * 3 * hidden * (4 * 1024 + 2 * hidden)
    return {"bytes": float(bytes_), "flops": float(flops)}


def _step_work(case):
    size = 2 if case["dtype"] == "bf16" else 4
    new, context, batch = lengths(case), case["context"], case["batch"]
    tokens = sum(new)
    if case["model"] == "llama":
        layer, kv, pair, state = 2048 * (3072 + 2048 + 3 * 8192), 1024, 32 * 128, [0]
        layers = [layer] * case["layers"]
        attention = case["layers"]
        states = 0
    else:
        delta = 2048 * (4 * 2048 + 32)
        mamba = 2048 * (2 * 4096 + 256 + 64 + 4096)
        both = 2048 * (3072 + 2048) + 2048 * (2 * 2048 + 128 + 32 + 2048)
        layers = [(delta, mamba, both)[i % 3] + 3 * 2048 * 8192 for i in range(case["layers"])]
        kv, pair = 1024, 32 * 128
        attention = sum(1 for i in range(case["layers"]) if i % 3 == 2)
        states = sum((16 * 128 * 128, 64 * 64 * 128, 32 * 64 * 64)[i % 3] for i in range(case["layers"]))
    wanted = sum(1 if context else len(_wanted(n)) for n in new)
    head = 2048 * 128256
    bytes_ = size * (sum(layers) + head + tokens * 2048) + 4 * wanted * 128256
    bytes_ += attention * size * kv * (batch * context + tokens) + 4 * batch * states * (2 if context else 1)
    flops = 2.0 * tokens * sum(layers) + 2.0 * wanted * head + 4.0 * tokens * states
    flops += attention * sum(2.0 * pair * (n * context + n * (n + 1) / 2) for n in new)
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    """About four times what the code of each kind was seen to differ from 64 bits by (the stream and the states of a layer are
    float32 sums over bfloat16 operands; logits have been through every layer's rounding)."""
    if case["kind"] == "step":
        return {"rel": 1e-4 if case["dtype"] == "fp32" else 0.03}
    # a router's close call falls the other way where its input's rounding differs: an expert of the token is another one then
    return {"rel": 0.03 if case["part"] == "moe" else 0.015}


# -------------------------------------------------------------------------------------------------------------- exact
# The same in float64, token by token, a function for each mechanism.

def _f64(tensors):
    return {k: v.double() for k, v in tensors.items()}


def _rms(x, eps, weight=None):
    y = x / (x.square().mean(-1, keepdim=True) + eps).sqrt()
    return y if weight is None else y * weight


def _layer_norm(x, eps, weight):
    x = x - x.mean(-1, keepdim=True)
    return _rms(x, eps, weight)


def _silu(x):
    return x * torch.sigmoid(x)


def _frequencies(dims, base):
    return base ** (-torch.arange(0, dims, 2, device=DEVICE, dtype=torch.float64) / dims)


def _llama3(freq, factor, low, high, original):
    wave = 2.0 * math.pi / freq
    smooth = (original / wave - low) / (high - low)
    out = torch.where(wave > original / low, freq / factor, (1.0 - smooth) * freq / factor + smooth * freq)
    return torch.where(wave < original / high, freq, out)


def _rotate(x, positions, freq, interleaved=False):
    """x [tokens, heads, dim]; the first 2 * len(freq) numbers of a head turn."""
    n = 2 * freq.numel()
    angle = positions[:, None, None].double() * freq
    c, s = angle.cos(), angle.sin()
    a, b = (x[..., 0:n:2], x[..., 1:n:2]) if interleaved else (x[..., :n // 2], x[..., n // 2:n])
    p, q = a * c - b * s, b * c + a * s
    turned = torch.stack((p, q), -1).flatten(-2) if interleaved else torch.cat((p, q), -1)
    return torch.cat((turned, x[..., n:]), -1)


def _conv(x, tail, weight, bias=None):
    """x [tokens, channels] behind tail [taps - 1, channels]: outputs, and the new tail."""
    rows = torch.cat((tail, x), 0)
    taps = weight.shape[1]
    out = sum(rows[j:j + x.shape[0]] * weight[:, j] for j in range(taps))
    return _silu(out if bias is None else out + bias), rows[rows.shape[0] - (taps - 1):]


def _attend(q, k, v, scale, before, sink=None, window=None):
    """q [new, heads, d], k [all, kv, d], v [all, kv, e], query i at place before + i."""
    heads, groups = q.shape[1], q.shape[1] // k.shape[1]
    place = before + torch.arange(q.shape[0], device=DEVICE)
    other = torch.arange(k.shape[0], device=DEVICE)
    hidden = other[None] > place[:, None]
    if window:
        hidden |= other[None] <= place[:, None] - window
    out = torch.empty((q.shape[0], heads, v.shape[2]), dtype=torch.float64, device=DEVICE)
    for h in range(heads):
        score = (q[:, h] @ k[:, h // groups].T * scale).masked_fill(hidden, -math.inf)
        if sink is not None:
            score = torch.cat((score, sink[h].expand(score.shape[0], 1)), 1)
        p = torch.softmax(score, -1)
        out[:, h] = p[:, :k.shape[0]] @ v[:, h // groups]
    return out


def _mamba2(x, w, heads, state, tail, p, n, prefix="", eps=EPS, names=None):
    """x [tokens, hidden] of one sequence; state [heads, p, n]."""
    g = lambda key: w[prefix + (names or {}).get(key, {"in": "in_proj.weight", "conv": "conv1d.weight", "conv_bias": "conv1d.bias",
                                                       "norm": "norm.weight", "out": "out_proj.weight"}.get(key, key))]
    inner = heads * p
    z, xbc, dt = (x @ g("in").T).split((inner, inner + 2 * n, heads), 1)
    xbc, tail = _conv(xbc, tail, g("conv"), g("conv_bias"))
    dt = torch.nn.functional.softplus(dt + g("dt_bias"))
    decay = torch.exp(-torch.exp(g("A_log")) * dt)
    xs, b, c = xbc[:, :inner].view(-1, heads, p), xbc[:, inner:inner + n], xbc[:, inner + n:]
    y = torch.empty_like(xs)
    for t in range(x.shape[0]):
        state = decay[t, :, None, None] * state + (dt[t, :, None] * xs[t])[:, :, None] * b[t]
        y[t] = state @ c[t]
    y = (y + g("D")[:, None] * xs).reshape(-1, inner) * _silu(z)
    return _rms(y, eps, g("norm")) @ g("out").T, state, tail


def _delta(x, w, heads, qk_heads, state, tail, d, e, prefix="", eps=EPS, names=None):
    """The gated delta rule; state [heads, e, d]."""
    names = names or {}
    g = lambda key: w[prefix + names.get(key, {"A_log": "A_log", "dt_bias": "dt_bias", "norm": "o_norm.weight", "out": "o_proj.weight", "q_conv": "q_conv1d.weight",
                                               "k_conv": "k_conv1d.weight", "v_conv": "v_conv1d.weight"}.get(key, key + "_proj.weight"))]
    qk = qk_heads * d
    made, tail = _conv(torch.cat([x @ g(key).T for key in ("q", "k", "v")], 1), tail, torch.cat([g(key + "_conv") for key in ("q", "k", "v")]))
    unit = lambda a: a / (a.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    share = heads // qk_heads
    q = (unit(made[:, :qk].view(-1, qk_heads, d)) * d ** -0.5).repeat_interleave(share, 1)
    k = unit(made[:, qk:2 * qk].view(-1, qk_heads, d)).repeat_interleave(share, 1)
    v = made[:, 2 * qk:].view(-1, heads, e)
    beta = torch.sigmoid(x @ g("b").T)
    decay = torch.exp(-torch.exp(g("A_log")) * torch.nn.functional.softplus(x @ g("a").T + g("dt_bias")))
    o = torch.empty_like(v)
    for t in range(x.shape[0]):
        state = decay[t, :, None, None] * state
        u = beta[t, :, None] * (v[t] - (state @ k[t, :, :, None])[..., 0])
        state = state + u[:, :, None] * k[t, :, None, :]
        o[t] = (state @ q[t, :, :, None])[..., 0]
    o = _rms(o, eps, g("norm")) * _silu(x @ g("g").T).view(-1, heads, e)
    return o.reshape(-1, heads * e) @ g("out").T, state, tail


def _linear_attention(x, w, heads, sizes, state):
    d, e = sizes["key_dim"], sizes["value_dim"]
    q, k, v = ((x @ w[key + "_proj.weight"].T).view(x.shape[0], heads, -1) for key in ("q", "k", "v"))
    if sizes.get("activation"):
        q, k, v = _silu(q), _silu(k), _silu(v)
    if sizes.get("position"):
        freq, place = _frequencies(d, sizes["position"].params["theta"]), torch.arange(x.shape[0], device=DEVICE)
        q, k = _rotate(q, place, freq), _rotate(k, place, freq)
    k = k * sizes.get("key_scale", 1.0)
    decay = torch.tensor(sizes["decay"], dtype=torch.float64, device=DEVICE)[:, None, None]
    o = torch.empty_like(v)
    for t in range(x.shape[0]):
        state = decay * state + v[t][:, :, None] * k[t][:, None, :]
        o[t] = (state @ q[t][:, :, None])[..., 0]
    gate = x @ w["g_proj.weight"].T
    if sizes["norm"] == "all":
        o = _rms(o.reshape(-1, heads * e), sizes["eps"], w["norm.weight"]) * torch.sigmoid(gate)
    else:
        o = _rms(o, sizes["eps"]).reshape(-1, heads * e) * _silu(gate)
    return o @ w["o_proj.weight"].T, state


def _differential(x, w, sizes):
    heads, kv, d, e = sizes["heads"], sizes["kv_heads"], sizes["dim"], sizes["value_dim"]
    n = x.shape[0]
    q, k, v = (x @ w[key + "_proj.weight"].T + w[key + "_proj.bias"] for key in ("q", "k", "v"))
    coef, every = sizes["q_gain"]
    gain = 1.0 + coef * torch.log(torch.floor((torch.arange(n, device=DEVICE, dtype=torch.float64) + 1) / every) + 1)
    q, k, v = q.view(n, heads, 2, d) * gain[:, None, None, None], k.view(n, kv, 2, d), v.view(n, kv, e)
    lam = torch.exp((w["lambda_q1"] * w["lambda_k1"]).sum()) - torch.exp((w["lambda_q2"] * w["lambda_k2"]).sum()) + sizes["diff"]
    first, second = (_attend(q[:, :, m], k[:, :, m], v, sizes["scale"], 0) for m in (0, 1))
    o = _rms(first - lam * second, sizes["eps"]) * (1.0 - sizes["diff"])
    return o.reshape(n, -1) @ w["o_proj.weight"].T


def _latent(x, w, sizes, past, context):
    """One token of one sequence: x [1, hidden], past [tokens, 576]."""
    heads, d, r, e, rank = sizes["heads"], sizes["dim"], sizes["rot_dim"], sizes["value_dim"], sizes["kv_rank"]
    place = torch.tensor([context], device=DEVICE)
    freq = _frequencies(r, sizes["position"].params["theta"])
    q = (_rms(x @ w["q_a_proj.weight"].T, sizes["eps"], w["q_a_norm.weight"]) @ w["q_b_proj.weight"].T).view(1, heads, d + r)
    q = torch.cat((q[..., :d], _rotate(q[..., d:], place, freq)), -1)
    made = x @ w["kv_a_proj.weight"].T
    row = torch.cat((_rms(made[:, :rank], sizes["eps"], w["kv_a_norm.weight"]), _rotate(made[:, None, rank:], place, freq)[:, 0]), 1)
    rows = torch.cat((past, row), 0)[-sizes["window"]:]
    c, shared = rows[:, :rank], rows[:, rank:]
    k = torch.cat(((c @ w["k_b_proj.weight"].T).view(-1, heads, d), shared[:, None].expand(-1, heads, r)), -1)
    v = (c @ w["v_b_proj.weight"].T).view(-1, heads, e)
    return _attend(q, k, v, sizes["scale"], rows.shape[0] - 1).reshape(1, -1) @ w["o_proj.weight"].T


def _moe(x, w, sizes):
    experts, groups = sizes["experts"], sizes["groups"]
    score = torch.softmax(x @ w["router.weight"].T, -1)
    best = score.view(-1, groups, experts // groups).amax(-1).topk(sizes["keep"], -1).indices
    allowed = torch.zeros((x.shape[0], groups), device=DEVICE).scatter_(1, best, 1.0).repeat_interleave(experts // groups, 1)
    value, chosen = score.masked_fill(allowed == 0, -1.0).topk(sizes["top"], -1)
    weight = torch.zeros_like(score).scatter_(1, chosen, value / (value.sum(-1, keepdim=True) + 1e-20))
    expert = lambda prefix: (_silu(x @ w[prefix + "gate_proj.weight"].T) * (x @ w[prefix + "up_proj.weight"].T)) @ w[prefix + "down_proj.weight"].T
    out = expert("shared.")
    for index in range(experts):
        out = out + weight[:, index:index + 1] * expert("experts.%d." % index)
    return out


def exact(case, seed):
    return _exact_step(case, seed) if case["kind"] == "step" else _exact_layer(case, seed)


def _exact_layer(case, seed):
    registry, kind, sizes = _part(case)
    part = registry.build(kind, sizes)
    w = _f64(_tensors(part.weights(), seed, torch.bfloat16))
    stream, norms, past, _ = _layer_inputs(case, part, seed)
    stream, norms, new, name, heads = stream.double(), [n.double() for n in norms], case["new"], case["part"], case["heads"]
    x = _rms(stream, EPS, norms[0])
    rows, kept = [], []
    zeros = lambda *shape: torch.zeros(shape, dtype=torch.float64, device=DEVICE)
    for i in range(case["batch"]):
        mine = x[i * new:(i + 1) * new]
        if name == "mamba2":
            y, state, tail = _mamba2(mine, w, heads, zeros(heads, 64, 128), zeros(3, heads * 64 + 256), 64, 128)
            kept.append((state, tail))
        elif name == "delta":
            y, state, tail = _delta(mine, w, heads, heads // 2, zeros(heads, 128, 128), zeros(3, 2 * heads * 128), 128, 128)
            kept.append((state, tail))
        elif name in ("lightning", "retention"):
            y, state = _linear_attention(mine, w, heads, sizes, zeros(heads, sizes["value_dim"], 128))
            kept.append((state,))
        elif name == "differential":
            y = _differential(mine, w, sizes)
        elif name == "latent":
            y = _latent(mine, w, sizes, past[i][0][0].double(), case["context"])
        else:
            y = _moe(mine, w, sizes)
        rows.append(y)
    stream = stream + torch.cat(rows, 0)
    return {"stream": stream, "normed": _rms(stream, EPS, norms[1]), "states": [torch.stack(s) for s in zip(*kept)]}


def _exact_step(case, seed):
    _, _, model = _model(case)
    w = _tensors(model.weight_declarations(), seed, DTYPES[case["dtype"]])
    tokens, past, states = _step_inputs(case, model, seed)
    lens, context = lengths(case), case["context"]
    llama = case["model"] == "llama"
    embed = w["model.embed_tokens.weight" if llama else "embed"]
    x = embed[torch.tensor(sum(tokens, []), device=DEVICE)].double()
    ends = torch.tensor([0] + lens, device="cpu").cumsum(0).tolist()
    spans = [slice(a, b) for a, b in zip(ends, ends[1:])]
    places = [context + torch.arange(n, device=DEVICE) for n in lens]
    entry = 0

    def attention(h, prefix, names, freq, interleaved, normed, entry):
        g = lambda key: w[prefix + names[key]].double()
        q, k, v = (h @ g(key).T for key in ("q", "k", "v"))
        q, k, v = q.view(-1, 32, 64), k.view(-1, 8, 64), v.view(-1, 8, 64)
        if normed:
            q, k = _rms(q, EPS, g("q_norm")), _rms(k, EPS, g("k_norm"))
        out = []
        for i, span in enumerate(spans):
            mine_q, mine_k = (_rotate(a[span], places[i], freq, interleaved) for a in (q, k))
            mine_v = v[span]
            if context:
                old_k, old_v = past[entry][i]
                mine_k, mine_v = torch.cat((old_k.double().transpose(0, 1), mine_k)), torch.cat((old_v.double().transpose(0, 1), mine_v))
            out.append(_attend(mine_q, mine_k, mine_v, 0.125, context, g("sink") if normed else None))
        return torch.cat(out).reshape(-1, 2048) @ g("o").T

    for layer in range(case["layers"]):
        if llama:
            p = "model.layers.%d." % layer
            h = _rms(x, 1e-5, w[p + "input_layernorm.weight"].double())
            s = LLAMA["rope_scaling"]
            freq = _llama3(_frequencies(64, 500000.0), s["factor"], s["low_freq_factor"], s["high_freq_factor"], s["original_max_position_embeddings"])
            x = x + attention(h, p + "self_attn.", {key: key + "_proj.weight" for key in "qkvo"}, freq, False, False, entry)
            entry += 1
            h = _rms(x, 1e-5, w[p + "post_attention_layernorm.weight"].double())
            gate, up, down = (w[p + "mlp.%s_proj.weight" % key].double() for key in ("gate", "up", "down"))
            x = x + (_silu(h @ gate.T) * (h @ up.T)) @ down.T
            continue
        p = "l%d." % layer
        h = _layer_norm(x, EPS, w[p + "norm1"].double())
        mixer = FAMALORN[layer % 3]["mixer"]
        mix = {k: v.double() for k, v in w.items() if k.startswith(p + "mix.")}
        mamba_names = {"in": "in", "conv": "conv", "conv_bias": "conv.b", "norm": "norm", "out": "o"}
        if layer % 3 == 0:
            names = {"q": "q", "k": "k", "v": "v", "q_conv": "q.conv", "k_conv": "k.conv", "v_conv": "v.conv", "b": "b", "a": "a", "g": "g", "norm": "norm", "out": "o"}
            add = torch.cat([_delta(h[s], mix, 16, 8, states[entry][0][i].double(), states[entry][1][i].double(), 128, 128, p + "mix.", EPS, names)[0]
                             for i, s in enumerate(spans)])
            entry += 1
        elif layer % 3 == 1:
            add = torch.cat([_mamba2(h[s], mix, 64, states[entry][0][i].double(), states[entry][1][i].double(), 64, 128, p + "mix.", EPS, mamba_names)[0]
                             for i, s in enumerate(spans)])
            entry += 1
        else:
            names = {"q": "q", "k": "k", "v": "v", "o": "o", "q_norm": "q.norm", "k_norm": "k.norm", "sink": "sink"}
            add = attention(h, p + "mix.left.", names, _frequencies(32, mixer["left"]["rot"]["base"]), True, True, entry)
            add = add + torch.cat([_mamba2(h[s], mix, 32, states[entry + 1][0][i].double(), states[entry + 1][1][i].double(), 64, 64, p + "mix.right.", EPS, mamba_names)[0]
                                   for i, s in enumerate(spans)])
            entry += 2
        x = x + add
        h = _layer_norm(x, EPS, w[p + "norm2"].double())
        gate, up, down = (w[p + "mlp." + key].double() for key in ("gate", "up", "down"))
        x = x + (torch.relu(h @ gate.T) * (h @ up.T)) @ down.T
    wanted = [span.start + place for span, n in zip(spans, lens) for place in ([0] if context else _wanted(n))]
    x = x[torch.tensor(wanted, device=DEVICE)]
    x = _rms(x, 1e-5, w["model.norm.weight"].double()) if llama else _layer_norm(x, EPS, w["final.norm"].double())
    return x @ (embed if llama else w["head"]).double().T
