"""The work that a program of this framework has it do, as cases that can be timed and compared: whole steps of the
engine (decoding and a prompt), and single layers of every kind that carries a served design (a dense decoder layer
over a large batch of long contexts and over a mixed step, attention over a long prompt, the true 32-bit path, the
recurrences with a matrix state, routed experts).  Every case goes through the entry points that a program calls:
`Engine.step`, or a layer's parts as they are built from a `PartSpec` and run on a step's batch.

Sizes are those of the benchmark's configurations.  Weights are random, of the scale that keeps a layer's output of the
order of its input; decays and forget gates are those of trained recurrences (a memory of tens to hundreds of tokens).
"""
import math

import torch

import tokenizer_b200 as tb
from tokenizer_b200.cache.device import DeviceCache
from tokenizer_b200.config import PartSpec
from tokenizer_b200.config.spec import LayerCall
from tokenizer_b200.engine.batch import BatchBuilder, StepEntry
from tokenizer_b200.kernels import ops
from tokenizer_b200.parts import DecoderModel, ResidualStream, Runtime, build_part, declared_tensors, part_class
from tokenizer_b200.weights import WeightStore

DEVICE = torch.device("cuda:0")
F64 = torch.float64
EPS = 1e-6
PAGE = 16

# hidden, query heads, key/value heads, lanes a head, feed-forward, layers
QWEN = {"0.5b": (896, 14, 2, 64, 4864, 24), "1.5b": (1536, 12, 2, 128, 8960, 28), "7b": (3584, 28, 4, 128, 18944, 28)}
VOCAB = 151936
# attention alone: hidden, query heads, key/value heads, lanes a head
ATTENTION = {"0.5b": (896, 14, 2, 64), "1k": (1024, 16, 4, 64), "2k": (2048, 16, 4, 128), "7b": (3584, 28, 4, 128)}
# recurrences and experts at the two widths
DELTA = {"1k": dict(hidden_size=1024, heads=8, kv_heads=4, dim=128, vdim=128, conv=4),
         "2k": dict(hidden_size=2048, heads=16, kv_heads=8, dim=128, vdim=128, conv=4)}
SPACE = {"1k": dict(hidden_size=1024, heads=16, vdim=64, state=128, groups=1, conv=4, norm_groups=1),
         "2k": dict(hidden_size=2048, heads=64, vdim=64, state=128, groups=8, conv=4, norm_groups=8)}
MEMORY = {"1k": dict(hidden_size=1024, heads=8, dim=64, vdim=128, gate_cap=15.0),
          "2k": dict(hidden_size=2048, heads=16, dim=128, vdim=128, gate_cap=15.0)}
EXPERTS = {"1k": dict(hidden_size=1024, experts=8, top=2, expert_inner=704, shared_inner=1408, activation="silu"),
           "2k": dict(hidden_size=2048, experts=8, top=2, expert_inner=1408, shared_inner=2816, activation="silu")}


def listed():
    return [
        # one user's chat: the smallest step there is, bound by latency and launches
        {"name": "decode_1", "kind": "step", "size": "0.5b", "requests": 1, "context": 512, "tokens": 1},
        # the benchmark's own decoding step: eight requests behind 512-token prompts
        {"name": "decode_8", "kind": "step", "size": "0.5b", "requests": 8, "context": 512, "tokens": 1},
        # a prompt that fills a step's token budget
        {"name": "prompt_2048", "kind": "step", "size": "0.5b", "requests": 1, "context": 0, "tokens": 2048},
        # a layer of a wide model while a full server decodes behind long, ragged contexts
        {"name": "decode_64_long", "kind": "layer", "size": "7b", "dtype": "bfloat16", "prompts": 0, "tokens": 0,
         "singles": 64, "context": 8192},
        # a layer in a busy scheduler's step: ragged portions of three prompts beside decoded tokens
        {"name": "mixed_step", "kind": "layer", "size": "1.5b", "dtype": "bfloat16", "prompts": 3, "tokens": 1900,
         "singles": 29, "context": 2048},
        # attention over one long document
        {"name": "attention_8192", "kind": "attention", "size": "7b", "prompts": 1, "tokens": 8192, "window": 0},
        # the true 32-bit path, as results are checked with it: a prompt of odd length
        {"name": "prompt_f32", "kind": "layer", "size": "0.5b", "dtype": "float32", "prompts": 1, "tokens": 777,
         "singles": 0, "context": 0},
        # the gated delta rule over a lone prompt (a chain of tokens)
        {"name": "delta_2048", "kind": "delta", "size": "2k", "prompts": 1, "tokens": 2048},
        # the delta rule with a decay a channel over four ragged prompts
        {"name": "channel_delta_4", "kind": "channel_delta", "size": "2k", "prompts": 4, "tokens": 5100},
        # the state-space recurrence over two ragged prompts
        {"name": "state_space_2", "kind": "state_space", "size": "2k", "prompts": 2, "tokens": 3001},
        # the matrix memory over a lone prompt
        {"name": "memory_2048", "kind": "memory", "size": "2k", "prompts": 1, "tokens": 2048},
        # routed experts with a shared one on a prompt's rows
        {"name": "experts_2048", "kind": "experts", "size": "2k", "prompts": 1, "tokens": 2048},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "layer", "layer", "attention", "f32", "delta", "channel_delta", "state_space",
                       "memory", "experts"])
    if kind == "step":
        if rng.random() < 0.5:
            return {"kind": "step", "size": "0.5b", "requests": _log(rng, 1, 32), "context": _log(rng, 64, 2000), "tokens": 1}
        return {"kind": "step", "size": "0.5b", "requests": 1, "context": 0, "tokens": _log(rng, 90, 2048)}
    if kind == "layer":
        size = rng.choice(["0.5b", "1.5b", "7b"])
        if rng.random() < 0.5:
            return {"kind": "layer", "size": size, "dtype": "bfloat16", "prompts": 0, "tokens": 0,
                    "singles": _log(rng, 1, 64), "context": _log(rng, 256, 8192)}
        return {"kind": "layer", "size": size, "dtype": "bfloat16", "prompts": rng.randint(1, 6),
                "tokens": _log(rng, 300, 2048 if size == "7b" else 4096), "singles": rng.randint(0, 31), "context": _log(rng, 64, 2048)}
    if kind == "f32":
        return {"kind": "layer", "size": "0.5b", "dtype": "float32", "prompts": 1, "tokens": _log(rng, 33, 1024),
                "singles": 0, "context": 0}
    if kind == "attention":
        return {"kind": "attention", "size": rng.choice(sorted(ATTENTION)), "prompts": rng.randint(1, 4),
                "tokens": _log(rng, 700, 8192), "window": rng.choice([0, 0, 1024])}
    return {"kind": kind, "size": rng.choice(["1k", "2k"]), "prompts": rng.randint(1, 4), "tokens": _log(rng, 300, 5100)}


# ---- a batch: which requests bring how many tokens behind how many ------------------------------------------------
def _ragged(total, parts):
    """`total` tokens over `parts` prompts of unlike lengths, each at least two."""
    weights = [1.0 + 0.37 * ((5 * i + 2) % 7) for i in range(parts)]
    lengths = [max(2, int(total * w / sum(weights))) for w in weights]
    lengths[-1] = max(2, lengths[-1] + total - sum(lengths))
    return lengths


def _batch(case):
    """[(tokens already held, new tokens)] of a layer's step, the portions first."""
    if case["kind"] == "step":
        return [(max(0, case["context"] - 3 * r), case["tokens"]) for r in range(case["requests"])]
    out = [(0, n) for n in _ragged(case["tokens"], case["prompts"])] if case["prompts"] else []
    singles = case.get("singles", 0)
    return out + [(max(1, case["context"] * (4 * singles - 3 * i) // (4 * singles)), 1) for i in range(singles)]


# ---- weights ------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed & 0x7FFFFFFF)


def _weights(specs, seed, whole=False):
    """name -> tensor, stored as released checkpoints are (bfloat16).  A matrix is drawn so that its products have the
    scale of its input (a whole model's: 0.02, as checkpoints begin); what sets a decay or a gate, as trained ones are."""
    out = {}
    for at, spec in enumerate(sorted(specs, key=lambda s: s.name)):
        shape = tuple(int(n) for n in spec.shape)
        value = torch.randn(shape, generator=_generator(seed * 1009 + at), device=DEVICE)
        if spec.name.endswith((".dt_bias",)):
            value = 0.5 * value - 3.5
        elif spec.name.endswith(".f.b"):
            value = 0.5 * value + 4.0
        elif spec.init == "one_plus_normal":
            value = 1.0 + 0.1 * value
        elif spec.std != 0.02 or len(shape) == 1:
            value = spec.std * value
        elif not whole:
            value = value / math.sqrt(shape[1])
            if spec.name.endswith((".q_proj.weight", ".q")):
                value = 2.0 * value                 # scores with a spread: some keys count, most do not
        elif "embed_tokens" in spec.name:
            value = 0.5 * value                     # a stream that every layer adds a little to, as in trained models
        else:
            value = 0.02 * value
        out[spec.name] = value.to(torch.bfloat16)
    return out


# ---- whole steps --------------------------------------------------------------------------------------------------
_kept = {}      # the engine of the step case at hand: a server keeps its model and engine over all its requests


def _step_config(size):
    hidden, nh, nkv, d, ff, layers = QWEN[size]
    return tb.Qwen2Config.from_dict({
        "architectures": ["Qwen2ForCausalLM"], "vocab_size": VOCAB, "hidden_size": hidden, "intermediate_size": ff,
        "num_hidden_layers": layers, "num_attention_heads": nh, "num_key_value_heads": nkv,
        "max_position_embeddings": 32768, "sliding_window": 32768, "max_window_layers": layers,
        "use_sliding_window": False, "tie_word_embeddings": True, "rope_theta": 1e6, "rms_norm_eps": EPS,
        "hidden_act": "silu"})


def _step_weights(size):
    return _weights(declared_tensors(_step_config(size).model_spec()), 7, whole=True)


def _step_engine(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _kept:
        _kept.clear()
        config = _step_config(case["size"])
        model = DecoderModel(config.model_spec(), WeightStore(_step_weights(case["size"])), Runtime(DEVICE, torch.bfloat16))
        pages = sum(-(-(held + new) // PAGE) for held, new in _batch(case))
        _kept[key] = tb.Engine(model, num_pages=6 * pages + 16, page_size=PAGE, max_requests=6 * case["requests"] + 2)
    return _kept[key]


def _step_tokens(case, seed):
    g = _generator(seed)
    return [torch.randint(0, VOCAB, (held + new,), generator=g, device=DEVICE).tolist() for held, new in _batch(case)]


class _Requests:
    """The requests of one state, closed with it."""

    def __init__(self, engine, names):
        self.engine, self.caches = engine, [engine.cache.open(n) for n in names]

    def __del__(self):
        for cache in self.caches:
            if not cache.closed:
                self.engine.cache.close(cache)


_names = iter(range(1 << 60))


def _prepare_step(case, seed):
    engine = _step_engine(case)
    tokens = _step_tokens(case, seed)
    if case["tokens"] > 1:
        return {"engine": engine, "tokens": tokens, "held": None}
    held = _Requests(engine, [("held", next(_names)) for _ in tokens])
    for cache, ids in zip(held.caches, tokens):
        engine.cache.reserve(cache, len(ids))
        if len(ids) > 1:
            engine.step([StepEntry(cache, ids[:-1], [])])
    return {"engine": engine, "tokens": tokens, "held": held}


def _run_step(state):
    engine, tokens = state["engine"], state["tokens"]
    if state["held"] is None:                    # a prompt: a request comes, its prompt runs, its pages go back
        entries = []
        for ids in tokens:
            cache = engine.cache.open(("prompt", next(_names)))
            engine.cache.reserve(cache, len(ids))
            entries.append(StepEntry(cache, ids, [len(ids) - 1]))
        logits = engine.step(entries)
        for e in entries:
            engine.cache.close(e.cache)
        return logits
    logits = engine.step([StepEntry(c, ids[-1:], [0]) for c, ids in zip(state["held"].caches, tokens)])
    for c in state["held"].caches:               # the token is taken back: a draft that was rejected
        c.length -= 1
    return logits


# ---- single layers ------------------------------------------------------------------------------------------------
def _layer_specs(case):
    """{name in the block: (category, PartSpec)} of a case's layer, the norms included."""
    kind = case["kind"]
    if kind == "layer":
        hidden, nh, nkv, d, ff, _ = QWEN[case["size"]]
        position = PartSpec("rope_half_split", {"theta": 1e6, "rotary_dim": d, "max_positions": 16384})
        return {"mixer_norm": ("norm", PartSpec("rms_norm", {"size": hidden, "eps": EPS}, "norm1")),
                "mixer": ("mixer", PartSpec("gqa_attention", {
                    "hidden_size": hidden, "num_heads": nh, "num_kv_heads": nkv, "head_dim": d, "qkv_bias": True,
                    "out_bias": False, "window": None, "position": position}, "attn")),
                "feed_forward_norm": ("norm", PartSpec("rms_norm", {"size": hidden, "eps": EPS}, "norm2")),
                "feed_forward": ("feed_forward", PartSpec("gated_mlp", {
                    "hidden_size": hidden, "intermediate_size": ff, "activation": "silu"}, "mlp"))}
    if kind == "attention":
        hidden, nh, nkv, d = ATTENTION[case["size"]]
        part = PartSpec("gqa_rotary", {
            "hidden_size": hidden, "heads": nh, "kv_heads": nkv, "dim": d, "vdim": d, "scale": d ** -0.5, "bias": True,
            "window": case["window"] or None, "position": PartSpec("rope_half", {"base": 1e6, "dims": d // 2})}, "attn")
    elif kind in ("delta", "channel_delta"):
        part = PartSpec("gated_delta_net" if kind == "delta" else "channel_delta_net", dict(DELTA[case["size"]], eps=EPS), "mix")
    elif kind == "state_space":
        part = PartSpec("mamba2", dict(SPACE[case["size"]], eps=EPS), "mix")
    elif kind == "memory":
        part = PartSpec("matrix_memory", dict(MEMORY[case["size"]], eps=EPS), "mix")
    else:
        part = PartSpec("routed_mlp", dict(EXPERTS[case["size"]]), "mlp")
    norm = PartSpec("rms_norm", {"size": part.params["hidden_size"], "eps": EPS}, "norm1")
    return {"mixer_norm": ("norm", norm), ("feed_forward" if kind == "experts" else "mixer"):
            ("feed_forward" if kind == "experts" else "mixer", part)}


def _layer_weights(case):
    specs = []
    for category, spec in _layer_specs(case).values():
        specs += part_class(category, spec.kind).tensors(spec)
    return _weights(specs, 3)


def _hidden(case):
    return next(s.params["size"] for c, s in _layer_specs(case).values() if c == "norm")


def _inputs(case, seed):
    """(the stream's rows; per request the keys and values it already holds)."""
    g = _generator(seed)
    batch = _batch(case)
    x = torch.randn((sum(new for _, new in batch), _hidden(case)), generator=g, device=DEVICE)
    past = []
    if case["kind"] == "layer":
        _, _, nkv, d, _, _ = QWEN[case["size"]]
        dtype = getattr(torch, case["dtype"])
        past = [torch.randn((2, held, nkv, d), generator=g, device=DEVICE).to(dtype) for held, _ in batch]
    return x, past


def _prepare_layer(case, seed):
    runtime = Runtime(DEVICE, getattr(torch, case.get("dtype", "bfloat16")))
    store = WeightStore(_layer_weights(case))
    built = {name: build_part(category, spec, store, runtime) for name, (category, spec) in _layer_specs(case).items()}
    x, past = _inputs(case, seed)
    state = {"x": x, "parts": built, "scratch": ops.ScratchSpace(), "ctx": None, "binding": None, "slots": None}
    mixer = built.get("mixer")
    if mixer is None:
        return state
    batch = _batch(case)
    need = mixer.cache_need()
    pages = sum(-(-(held + new) // PAGE) for held, new in batch) if need.kv is not None else 1
    cache = DeviceCache([need], pages, PAGE, len(batch), runtime)
    binding = cache.bindings([LayerCall(0)])[0]
    notes = getattr(mixer, "batch_annotations", lambda: [])()
    builder = BatchBuilder(cache, 2, 1 << 24, DEVICE, notes)
    entries = []
    for r, (held, new) in enumerate(batch):
        request = cache.open(r)
        cache.reserve(request, held + new)
        if held:
            at = torch.arange(held, device=DEVICE)
            pages_of = torch.tensor(request.tables[0], device=DEVICE)
            rows = pages_of[at // PAGE] * PAGE + at % PAGE
            binding.k_pool[rows] = past[r][0]
            binding.v_pool[rows] = past[r][1]
            cache.commit(request, held)
        entries.append(StepEntry(request, [0] * new, []))
    state["ctx"], _, _ = builder.build(entries)
    state.update(binding=binding, cache=cache, builder=builder)
    if case["kind"] == "layer":
        state["block"] = part_class("block", "pre_norm_residual")(**built)
    else:
        state["block"] = part_class("block", "pre_norm_mixer_only")(**built)
    # the recurrences' matrices, as the request's slots hold them
    if binding.state is not None:
        state["matrices"] = binding.state[:len(batch), :_matrix_floats(case)]
    return state


def _run_layer(state):
    with ops.bound_stream(), ops.scratch_scope(state["scratch"]):
        stream = ResidualStream(state["x"].clone())
        if state["binding"] is None:             # a feed-forward alone
            stream.add(state["parts"]["feed_forward"].forward(stream.normed(state["parts"]["mixer_norm"])))
        else:
            state["block"].forward(stream, state["ctx"], state["binding"])
        out = stream.flush()
    return {"x": out, "state": state["matrices"]} if "matrices" in state else {"x": out}


def prepare(case, seed):
    with torch.no_grad():
        return _prepare_step(case, seed) if case["kind"] == "step" else _prepare_layer(case, seed)


def run(state):
    return _run_step(state) if "engine" in state else _run_layer(state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _matrix_floats(case):
    """Floats of a request's matrices in its slot (the recurrences')."""
    if case["kind"] in ("delta", "channel_delta"):
        p = DELTA[case["size"]]
        return p["heads"] * p["vdim"] * p["dim"]
    if case["kind"] == "state_space":
        p = SPACE[case["size"]]
        return p["heads"] * p["vdim"] * p["state"]
    p = MEMORY[case["size"]]
    return p["heads"] * (p["vdim"] + 1) * p["dim"]


def _seen(held, new, window):
    """Pairs of a query and a key that it sees."""
    return sum(min(held + i + 1, window + 1) if window else held + i + 1 for i in range(new))


def work(case):
    batch, kind = _batch(case), case["kind"]
    rows = sum(new for _, new in batch)
    pairs = sum(_seen(held, new, case.get("window", 0)) for held, new in batch)
    keys = sum(held + new for held, new in batch)
    if kind in ("step", "layer"):
        hidden, nh, nkv, d, ff, layers = QWEN[case["size"]]
        layers = layers if kind == "step" else 1
        size = 4 if case.get("dtype") == "float32" else 2
        matrix = hidden * (nh + 2 * nkv) * d + nh * d * hidden + 3 * hidden * ff
        flops = layers * (2.0 * rows * matrix + 4.0 * pairs * nh * d)
        moved = layers * (matrix * size + 2.0 * keys * nkv * d * size)
        if kind == "step":
            wanted = len(batch)
            flops += 2.0 * wanted * hidden * VOCAB
            moved += VOCAB * hidden * 2 + wanted * VOCAB * 4
        else:
            moved += rows * hidden * 8
        return {"bytes": moved, "flops": flops}
    if kind == "attention":
        hidden, nh, nkv, d = ATTENTION[case["size"]]
        matrix = hidden * (2 * nh + 2 * nkv) * d
        return {"bytes": matrix * 2.0 + rows * hidden * 8.0 + 4.0 * rows * nkv * d,
                "flops": 2.0 * rows * matrix + 4.0 * pairs * nh * d}
    if kind == "experts":
        p = EXPERTS[case["size"]]
        used = 3 * p["hidden_size"] * (p["top"] * p["expert_inner"] + p["shared_inner"])
        held = 3 * p["hidden_size"] * (p["experts"] * p["expert_inner"] + p["shared_inner"])
        return {"bytes": held * 2.0 + rows * p["hidden_size"] * 8.0, "flops": 2.0 * rows * used}
    floats = _matrix_floats(case)
    if kind in ("delta", "channel_delta"):
        p = DELTA[case["size"]]
        per_token = 2 * p["kv_heads"] * p["dim"] + 2 * p["heads"] * p["vdim"] + 2 * p["heads"]
        steps = 8.0
    elif kind == "state_space":
        p = SPACE[case["size"]]
        per_token = 2 * p["heads"] * p["vdim"] + 2 * p["groups"] * p["state"] + p["heads"]
        steps = 6.0
    else:
        p = MEMORY[case["size"]]
        per_token = p["heads"] * (2 * p["dim"] + 2 * p["vdim"] + 2)
        steps = 6.0
    matrix = p["hidden_size"] * (per_token + p["heads"] * p["vdim"])
    return {"bytes": matrix * 2.0 + rows * p["hidden_size"] * 8.0 + 8.0 * floats * len(batch),
            "flops": 2.0 * rows * matrix + steps * rows * floats}


def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    if case["kind"] == "step":
        return {"rel": 2e-2, "max": 0.3}
    if case["kind"] == "experts":                   # a close call between two experts moves a whole row
        return {"rel": 2e-2, "max": 0.99}
    return {"rel": 1e-2, "max": 0.3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _rms(x, gain, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _turn(x, positions, theta, dims):
    """The half layout of the rotation on the first `dims` lanes; angles are products of 32-bit numbers."""
    inv = torch.tensor([theta ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=F64, device=DEVICE)
    angle = (positions.to(torch.float32)[:, None] * inv.to(torch.float32)[None, :]).to(F64)
    cos, sin = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    u, v, rest = x[..., :dims // 2], x[..., dims // 2:dims], x[..., dims:]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, rest], dim=-1)


def _attend(q, k, v, held, window, scale):
    """[rows, heads, d] over the keys of one request, in pieces of rows."""
    rows, nh, d = q.shape
    share = nh // k.shape[1]
    out = torch.empty_like(q)
    at = torch.arange(k.shape[0], device=DEVICE)
    for first in range(0, rows, 2048):
        place = torch.arange(held + first, held + min(first + 2048, rows), device=DEVICE)
        hidden = at[None, :] > place[:, None]
        if window:
            hidden |= at[None, :] + window < place[:, None]
        for h in range(nh):
            s = (q[first:first + 2048, h] @ k[:, h // share].t()) * scale
            out[first:first + 2048, h] = torch.softmax(s.masked_fill(hidden, -math.inf), dim=-1) @ v[:, h // share]
    return out


def _qwen_layer(x, batch, past, w, names, sizes):
    """One dense decoder layer; `names` are the prefixes of its parts."""
    hidden, nh, nkv, d, _, _ = sizes
    norm1, attn, norm2, mlp = names

    def get(name):
        return w[name].to(F64)

    h = _rms(x, get(norm1 + ".weight"))
    q, k, v = (h @ get(f"{attn}.{n}_proj.weight").t() + get(f"{attn}.{n}_proj.bias") for n in "qkv")
    q, k, v = q.view(-1, nh, d), k.view(-1, nkv, d), v.view(-1, nkv, d)
    mixed, row = torch.empty_like(q), 0
    for r, (held, new) in enumerate(batch):
        positions = torch.arange(held, held + new, device=DEVICE)
        rows = slice(row, row + new)
        keys, values = _turn(k[rows], positions, 1e6, d), v[rows]
        if held:
            keys, values = torch.cat([past[r][0].to(F64), keys]), torch.cat([past[r][1].to(F64), values])
        mixed[rows] = _attend(_turn(q[rows], positions, 1e6, d), keys, values, held, 0, d ** -0.5)
        row += new
    x = x + mixed.reshape(-1, nh * d) @ get(attn + ".o_proj.weight").t()
    h = _rms(x, get(norm2 + ".weight"))
    gate = h @ get(mlp + ".gate_proj.weight").t()
    inner = gate * torch.sigmoid(gate) * (h @ get(mlp + ".up_proj.weight").t())
    return x + inner @ get(mlp + ".down_proj.weight").t()


def _exact_step(case, seed):
    batch = [(0, held + new) for held, new in _batch(case)]
    if sum(n for _, n in batch) > 20000:
        return None
    w, tokens = _step_weights(case["size"]), _step_tokens(case, seed)
    sizes = QWEN[case["size"]]
    table = w["model.embed_tokens.weight"]
    x = table[torch.tensor([t for ids in tokens for t in ids], device=DEVICE)].to(F64)
    for i in range(sizes[5]):
        p = f"model.layers.{i}"
        x = _qwen_layer(x, batch, None, w, (p + ".input_layernorm", p + ".self_attn", p + ".post_attention_layernorm",
                                            p + ".mlp"), sizes)
    last = torch.tensor([sum(n for _, n in batch[:r + 1]) - 1 for r in range(len(batch))], device=DEVICE)
    return _rms(x[last], w["model.norm.weight"].to(F64)) @ table.to(F64).t()


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, taps, bias, batch):
    """The short causal convolution, channel by channel, zeros before a sequence's start, and silu."""
    out, row, n = torch.empty_like(x), 0, taps.shape[1]
    for _, new in batch:
        part = torch.cat([torch.zeros((n - 1, x.shape[1]), dtype=F64, device=DEVICE), x[row:row + new]])
        out[row:row + new] = sum(part[j:j + new] * taps[:, j] for j in range(n)) + (0 if bias is None else bias)
        row += new
    return _silu(out)


def _unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def _delta(h, batch, w, p, by_channel):
    heads, groups, dim, vdim = p["heads"], p["kv_heads"], p["dim"], p["vdim"]
    rows, share = h.shape[0], heads // groups

    def get(name):
        return w["mix." + name].to(F64)

    q, k, v = (_conv(h @ get(n).t(), get(n + ".conv"), None, batch) for n in "qkv")
    q = _unit(q.view(rows, groups, dim)).repeat_interleave(share, 1) * dim ** -0.5
    k = _unit(k.view(rows, groups, dim)).repeat_interleave(share, 1)
    v, beta = v.view(rows, heads, vdim), torch.sigmoid(h @ get("b").t())
    softplus = torch.nn.functional.softplus
    if by_channel:
        pre = (h @ get("a1").t()) @ get("a2").t() + get("dt_bias")
        decay = torch.exp(-torch.exp(get("A_log"))[:, None] * softplus(pre).view(rows, heads, dim))[..., None]
        gate = torch.sigmoid((h @ get("g1").t()) @ get("g2").t())
    else:
        decay = torch.exp(-torch.exp(get("A_log")) * softplus(h @ get("a").t() + get("dt_bias")))[..., None, None]
        gate = _silu(h @ get("g").t())
    o, states, row = torch.empty_like(v), [], 0
    for _, new in batch:
        s = torch.zeros((heads, dim, vdim), dtype=F64, device=DEVICE)
        for t in range(row, row + new):
            s = decay[t] * s
            u = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", s, k[t]))
            s = s + k[t][:, :, None] * u[:, None, :]
            o[t] = torch.einsum("hkv,hk->hv", s, q[t])
        states.append(s.transpose(1, 2).reshape(-1))
        row += new
    y = _rms(o, get("norm")).reshape(rows, -1) * gate
    return y @ get("o").t(), torch.stack(states)


def _state_space(h, batch, w, p):
    heads, vdim, n, groups = p["heads"], p["vdim"], p["state"], p["groups"]
    rows, inner, share = h.shape[0], heads * vdim, heads // groups

    def get(name):
        return w["mix." + name].to(F64)

    z, xbc, dt = torch.split(h @ get("in").t(), [inner, inner + 2 * groups * n, heads], dim=1)
    x, b, c = torch.split(_conv(xbc, get("conv"), get("conv.b"), batch), [inner, groups * n, groups * n], dim=1)
    x = x.view(rows, heads, vdim)
    b, c = (t.reshape(rows, groups, n).repeat_interleave(share, 1) for t in (b, c))
    dt = torch.nn.functional.softplus(dt + get("dt_bias"))
    decay = torch.exp(-torch.exp(get("A_log")) * dt)[..., None, None]
    y, states, row = torch.empty_like(x), [], 0
    for _, new in batch:
        s = torch.zeros((heads, n, vdim), dtype=F64, device=DEVICE)
        for t in range(row, row + new):
            s = decay[t] * s + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None, :]
            y[t] = torch.einsum("hnv,hn->hv", s, c[t])
        states.append(s.transpose(1, 2).reshape(-1))
        row += new
    y = (y + get("D")[:, None] * x).reshape(rows, inner) * _silu(z)
    parts = y.view(rows, p["norm_groups"], -1)
    y = (parts / torch.sqrt((parts * parts).mean(-1, keepdim=True) + EPS)).reshape(rows, inner) * get("norm")
    return y @ get("o").t(), torch.stack(states)


def _memory(h, batch, w, p):
    heads, dim, vdim, cap = p["heads"], p["dim"], p["vdim"], p["gate_cap"]
    rows = h.shape[0]

    def get(name):
        return w["mix." + name].to(F64)

    q = (h @ get("q").t()).view(rows, heads, dim) * dim ** -0.5
    k, v = (h @ get("k").t()).view(rows, heads, dim), (h @ get("v").t()).view(rows, heads, vdim)
    gate_in = cap * torch.tanh((h @ get("i").t() + get("i.b")) / cap)
    gate_f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ get("f").t() + get("f.b")) / cap))
    v = torch.cat([v, torch.ones((rows, heads, 1), dtype=F64, device=DEVICE)], dim=-1)      # n behind the columns
    o, states, row = torch.empty((rows, heads, vdim), dtype=F64, device=DEVICE), [], 0
    for _, new in batch:
        s = torch.zeros((heads, dim, vdim + 1), dtype=F64, device=DEVICE)
        m = torch.zeros(heads, dtype=F64, device=DEVICE)
        for t in range(row, row + new):
            top = torch.maximum(gate_f[t] + m, gate_in[t])
            s = torch.exp(gate_f[t] + m - top)[:, None, None] * s + \
                torch.exp(gate_in[t] - top)[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            m = top
            both = torch.einsum("hkv,hk->hv", s, q[t])
            o[t] = both[:, :vdim] / (torch.maximum(both[:, vdim].abs(), torch.exp(-m)) + 1e-6)[:, None]
        states.append(s.transpose(1, 2).reshape(-1))
        row += new
    y = _rms(o, 1.0).reshape(rows, -1) * get("norm") * torch.sigmoid(h @ get("g").t())
    return y @ get("o").t(), torch.stack(states)


def _experts(h, w, p):
    def get(name):
        return w["mlp." + name].to(F64)

    # the choice is made on what the layer reads, a row in bfloat16: a close call is settled there
    scores = h.to(torch.bfloat16).to(F64) @ get("router").t()
    best, chosen = torch.topk(scores, p["top"], dim=1)
    share = torch.zeros_like(scores).scatter_(1, chosen, torch.softmax(best, dim=1))
    out = torch.sigmoid(h @ get("shared.sg").t()) * (
        (_silu(h @ get("shared.gate").t()) * (h @ get("shared.up").t())) @ get("shared.down").t())
    for e in range(p["experts"]):
        inner = _silu(h @ get(f"e{e}.gate").t()) * (h @ get(f"e{e}.up").t())
        out = out + share[:, e:e + 1] * (inner @ get(f"e{e}.down").t())
    return out


def exact(case, seed):
    if case["kind"] == "step":
        return _exact_step(case, seed)
    w, batch = _layer_weights(case), _batch(case)
    x, past = _inputs(case, seed)
    x = x.to(F64)
    if case["kind"] == "layer":
        return {"x": _qwen_layer(x, batch, past, w, ("norm1", "attn", "norm2", "mlp"), QWEN[case["size"]])}
    h = _rms(x, w["norm1.weight"].to(F64))
    if case["kind"] == "attention":
        _, nh, nkv, d = ATTENTION[case["size"]]
        q, k, v = (h @ w["attn." + n].to(F64).t() + w[f"attn.{n}.b"].to(F64) for n in "qkv")
        q, k, v = q.view(-1, nh, d), k.view(-1, nkv, d), v.view(-1, nkv, d)
        mixed, row = torch.empty_like(q), 0
        for _, new in batch:
            positions, rows = torch.arange(new, device=DEVICE), slice(row, row + new)
            mixed[rows] = _attend(_turn(q[rows], positions, 1e6, d // 2), _turn(k[rows], positions, 1e6, d // 2), v[rows],
                                  0, case["window"], d ** -0.5)
            row += new
        return {"x": x + mixed.reshape(-1, nh * d) @ w["attn.o"].to(F64).t()}
    if case["kind"] == "experts":
        return {"x": x + _experts(h, w, EXPERTS[case["size"]])}
    if case["kind"] == "state_space":
        y, state = _state_space(h, batch, w, SPACE[case["size"]])
    elif case["kind"] == "memory":
        y, state = _memory(h, batch, w, MEMORY[case["size"]])
    else:
        y, state = _delta(h, batch, w, DELTA[case["size"]], case["kind"] == "channel_delta")
    return {"x": x + y, "state": state}
