"""The engine's everyday work as timed cases: decode and prefill steps of a whole model, and single layers of the other
architectures at their benchmark sizes, each through the call that a program makes.

Whole models run through ``ModelRunner`` (the step function), single layers through the registered part's ``forward`` on a
paged cache or a state slot.  Weights have the random-weights mode's distributions, made on the device.  Sizes are those of the
benchmark's shapes (``bench.py``): the Qwen2.5-0.5B shape, and the `1b` and `0.3b` shapes of the other architectures.

Kinds of case:

* ``decode``: one decode step of the 0.5B model, a token per request, through ``step_and_sample`` (a replayed graph); logits.
* ``prefill``: one step that runs whole prompts through the 0.5B model (``step``), logits at every prompt's last place.
* ``float32``: the same in the true 32-bit path, four layers and the head.
* ``map_attention``: a ``multimap_attention`` layer (differential attention; windows, sinks, capped scores, gates) over prompt
  portions, or one token per request over long contexts.
* ``latent_attention``: a ``latent_attention`` layer over prompt portions.
* ``experts``: a ``routed_experts`` layer.
* ``linear_attention``: a ``gated_linear_attention`` layer over new requests' prompts.
"""
import hashlib
import math
import random

import torch

from sprout_lm_b200 import ModelRunner, parse_config
from sprout_lm_b200.config.specs import PartSpec
from sprout_lm_b200.engine.batch import StepContext, StepEntry
from sprout_lm_b200.models import DecoderModel
from sprout_lm_b200.parts import CacheView, Runtime, StateView, WeightSource, build_part

DEVICE = "cuda:0"
PAGE = 16

QWEN_05B = {"architectures": ["Qwen2ForCausalLM"], "model_type": "qwen2", "hidden_act": "silu", "hidden_size": 896,
            "intermediate_size": 4864, "num_hidden_layers": 24, "num_attention_heads": 14, "num_key_value_heads": 2,
            "vocab_size": 151936, "max_position_embeddings": 4096, "rms_norm_eps": 1e-6, "rope_theta": 1000000.0,
            "tie_word_embeddings": True, "eos_token_id": 151645, "use_sliding_window": False, "rope_scaling": None}

# layers of the other architectures: the 1b shape, and the 0.3b shape of half its width and heads
SHAPES = {
    "1b": dict(width=2048, heads=16, kv_heads=4, kv_rank=512, q_rank=768, experts=32, identity=4, expert_ff=1024, shared_ff=2048,
               window=1024, state_heads=16, rank=32),
    "0.3b": dict(width=1024, heads=8, kv_heads=2, kv_rank=256, q_rank=384, experts=16, identity=2, expert_ff=512, shared_ff=1024,
                 window=512, state_heads=8, rank=16),
}
TOP, LIMIT, ALPHA = 4, 7.0, 1.702          # routed experts: taken per token, the gated activation's clamp and slope
STATE_DIM, TAU = 128, 16.0                 # gated linear attention: state of 128 x 128 per head
EPS = 1e-5


def listed():
    return [
        # one user waiting for the next token: the smallest call, a chain of dependent launches
        {"name": "decode-1", "kind": "decode", "requests": 1, "context": 512},
        # a small serving batch
        {"name": "decode-8", "kind": "decode", "requests": 8, "context": 600},
        # a busy server's batch over longer contexts
        {"name": "decode-64", "kind": "decode", "requests": 64, "context": 1500},
        # a long prompt, or a full portion of several in chunked prefill
        {"name": "prefill-2048", "kind": "prefill", "requests": 1, "tokens": 2048},
        # differential attention (two softmax maps per head) reading a prompt
        {"name": "two-map-prefill", "kind": "map_attention", "shape": "1b", "maps": 2, "dim": 64, "mask": "none", "softcap": 0.0,
         "extras": False, "requests": 1, "new": 2048, "held": 0},
        # sliding-window attention with a gate, several prompts of odd lengths in one step, continuing what is cached
        {"name": "window-prefill-ragged", "kind": "map_attention", "shape": "1b", "maps": 1, "dim": 64, "mask": "window",
         "softcap": 0.0, "extras": False, "requests": 5, "new": 4001, "held": 700},
        # softmax attention with capped scores, sinks and gates: a decode batch over long contexts
        {"name": "capped-decode-64", "kind": "map_attention", "shape": "1b", "maps": 1, "dim": 128, "mask": "none", "softcap": 30.0,
         "extras": True, "requests": 64, "new": 64, "held": 6000},
        # attention over a low-rank latent reading a prompt
        {"name": "latent-prefill", "kind": "latent_attention", "shape": "1b", "requests": 1, "new": 2048, "held": 0},
        # routed experts over a prompt: a contraction per expert
        {"name": "experts-2048", "kind": "experts", "shape": "1b", "tokens": 2048},
        # routed experts in a decode batch: a stream of the experts' weights
        {"name": "experts-64", "kind": "experts", "shape": "1b", "tokens": 64},
        # gated linear attention over the prompts of three new requests
        {"name": "linear-attention-ragged", "kind": "linear_attention", "shape": "1b", "requests": 3, "tokens": 2500},
        # the 32-bit path: a prompt through four layers
        {"name": "float32-prefill", "kind": "float32", "requests": 1, "tokens": 512},
    ]


def _spread(rng, low, high):
    """A whole number between the two, even over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "map_attention", "map_attention", "map_decode", "latent_attention", "experts",
                       "experts", "linear_attention", "float32"])
    shape = rng.choice(["1b", "0.3b"])
    if kind == "decode":
        return {"kind": kind, "requests": _spread(rng, 1, 64), "context": _spread(rng, 32, 1500)}
    if kind == "prefill":
        requests = rng.randint(1, 6)
        return {"kind": kind, "requests": requests, "tokens": _spread(rng, max(64, 8 * requests), 2048)}
    if kind == "float32":
        requests = rng.randint(1, 4)
        return {"kind": kind, "requests": requests, "tokens": _spread(rng, max(16, 4 * requests), 512)}
    if kind in ("map_attention", "map_decode"):
        maps = rng.choice([1, 1, 2])
        case = {"kind": "map_attention", "shape": shape, "maps": maps, "dim": 64 if maps == 2 else rng.choice([64, 128]),
                "mask": rng.choice(["none", "window"]) if maps == 1 else "none",
                "softcap": rng.choice([0.0, 30.0]) if maps == 1 else 0.0, "extras": maps == 1 and rng.random() < 0.5}
        if kind == "map_decode":
            requests = _spread(rng, 8, 64)
            return {**case, "requests": requests, "new": requests, "held": _spread(rng, 256, 6000)}
        requests = rng.randint(1, 6)
        return {**case, "requests": requests, "new": _spread(rng, 40 * requests, 2048), "held": rng.choice([0, _spread(rng, 16, 1024)])}
    if kind == "latent_attention":
        requests = rng.randint(1, 5)
        return {"kind": kind, "shape": shape, "requests": requests, "new": _spread(rng, 40 * requests, 2048),
                "held": rng.choice([0, _spread(rng, 16, 512)])}
    if kind == "experts":
        return {"kind": kind, "shape": shape, "tokens": _spread(rng, 8, 2048)}
    requests = rng.randint(1, 6)
    return {"kind": "linear_attention", "shape": shape, "requests": requests, "tokens": _spread(rng, 40 * requests, 2500)}


# ------------------------------------------------------------------ what a case consists of
def _lengths(total, parts):
    """``total`` split into ``parts`` uneven positive whole numbers, the same for every seed."""
    rng = random.Random(total * 64 + parts)
    weights = [rng.uniform(0.4, 1.6) for _ in range(parts)]
    lengths = [max(1, int(total * w / sum(weights))) for w in weights]
    lengths[0] += total - sum(lengths)
    return lengths


def _contexts(longest, requests):
    """What each request of a decode step holds: between half of the longest and the longest."""
    rng = random.Random(longest * 64 + requests)
    return [longest] + [rng.randint(max(1, longest // 2), longest) for _ in range(requests - 1)]


def _generator(seed, name):
    digest = hashlib.sha256(f"{seed}:{name}".encode()).digest()
    return torch.Generator(device=DEVICE).manual_seed(int.from_bytes(digest[:7], "little"))


def _normal(seed, name, shape, std=1.0, dtype=torch.float32):
    return (torch.randn(tuple(shape), generator=_generator(seed, name), device=DEVICE, dtype=torch.float32) * std).to(dtype)


def _weight(seed, name, shape, init):
    """A tensor with the random-weights mode's distribution; matrices rounded to bfloat16 as stored ones are."""
    values = _normal(seed, name, shape, 0.02)
    if init == "gain":
        return values + 1.0
    if init == "wide":
        return values * 10.0
    if init == "matrix":
        return values.to(torch.bfloat16)
    return values


class _Weights:
    """Random weights in the place of a model folder's tensors."""

    def __init__(self, decls, seed):
        self.decls, self.seed = {decl.name: decl for decl in decls}, seed

    def check(self, expected, ignorable=()):
        pass

    def tensor(self, name, shape=None):
        decl = self.decls[name]
        return _weight(self.seed, name, decl.shape, decl.init)


class _Exact:
    """The same weights as float64."""

    def __init__(self, seed):
        self.seed = seed

    def __call__(self, name, *shape, init="matrix"):
        return _weight(self.seed, name, shape, init).double()


def _model(case, seed):
    config = dict(QWEN_05B)
    dtype = torch.bfloat16
    if case["kind"] == "float32":
        config["num_hidden_layers"], dtype = 4, torch.float32
    model = DecoderModel(parse_config(config).model_spec())
    model.load(_Weights(model.tensor_decls(), seed), Runtime(DEVICE, dtype))
    return model


def _tokens(seed, counts):
    flat = torch.randint(0, QWEN_05B["vocab_size"], (sum(counts),), generator=_generator(seed, "tokens"), device=DEVICE).tolist()
    out, at = [], 0
    for n in counts:
        out.append(flat[at:at + n])
        at += n
    return out


def _held_rows(seed, name, counts, heads, width):
    """What the cache holds of each request before the pass: [held, heads, width] per request."""
    flat = _normal(seed, name, (sum(counts), heads, width), 0.6, torch.bfloat16)
    return list(flat.split(counts))


def _step_context(new, held, seed):
    """The batch of a step on the device: ``new`` tokens per request behind ``held`` cached ones, pages scattered over the pool."""
    requests, tokens = len(new), sum(new)
    total = [h + n for h, n in zip(held, new)]
    pages = [-(-t // PAGE) for t in total]
    order = torch.randperm(sum(pages), generator=_generator(seed, "pages"), device=DEVICE).to(torch.int32)
    table = torch.full((requests, -(-max(pages) // 64) * 64), -1, dtype=torch.int32, device=DEVICE)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n

    def ints(values):
        return torch.tensor(values, dtype=torch.int32).to(DEVICE)
    starts = [0]
    for n in new:
        starts.append(starts[-1] + n)
    empty = torch.zeros(tokens, dtype=torch.int32, device=DEVICE)
    return StepContext(
        num_tokens=tokens, num_seqs=requests, max_q_len=max(new), max_context=max(total), token_ids=empty,
        positions=ints([h + j for h, n in zip(held, new) for j in range(n)]),
        seq_of_token=ints([i for i, n in enumerate(new) for _ in range(n)]), q_start=ints(starts), context_lens=ints(total),
        state_slots=ints(list(range(requests))), logits_rows=ints([s - 1 for s in starts[1:]]), block_tables=[table],
        page_tokens=PAGE), sum(pages)


def _place(pool, table, rows):
    """Rows [held, heads, width] of every request into the pool's pages [pages, heads, PAGE, width]."""
    for i, part in enumerate(rows):
        n = part.shape[0]
        if n == 0:
            continue
        place = torch.arange(n, device=pool.device)
        pool[table[i].long()[place // PAGE], :, place % PAGE] = part.to(pool.dtype)


def _attention_case(case):
    if case["new"] == case["requests"]:
        held = _contexts(case["held"], case["requests"])
        return [1] * case["requests"], held
    return _lengths(case["new"], case["requests"]), [case["held"]] * case["requests"]


def _map_spec(case):
    z = SHAPES[case["shape"]]
    return PartSpec("multimap_attention", {
        "hidden_size": z["width"], "heads": z["heads"], "kv_heads": z["kv_heads"], "dim": case["dim"], "value_dim": 128,
        "scale": case["dim"] ** -0.5, "maps": case["maps"], "diff": 0.5 if case["maps"] == 2 else 0.0,
        "norm_eps": EPS if case["maps"] == 2 else 0.0, "out_scale": 0.5 if case["maps"] == 2 else 1.0,
        "position": PartSpec("rope_linear", {"dims": 64, "theta": 10000.0, "max_positions": 16384}),
        "mask": ("window", z["window"]) if case["mask"] == "window" else None, "softcap": case["softcap"],
        "sink": case["extras"], "gate": case["extras"] or case["mask"] == "window"})


def _latent_spec(case):
    z = SHAPES[case["shape"]]
    return PartSpec("latent_attention", {
        "hidden_size": z["width"], "heads": z["heads"], "dim": 64, "rot_dim": 64, "value_dim": 128, "kv_rank": z["kv_rank"],
        "q_rank": z["q_rank"], "scale": 128 ** -0.5, "eps": EPS,
        "position": PartSpec("rope_interleaved", {"dims": 64, "theta": 10000.0, "max_positions": 16384})})


def _expert_spec(case):
    z = SHAPES[case["shape"]]
    return PartSpec("routed_experts", {
        "hidden_size": z["width"], "experts": z["experts"], "identity": z["identity"], "top": TOP, "scale": 1.0,
        "expert_ff": z["expert_ff"], "expert_limit": LIMIT, "alpha": ALPHA, "shared_ff": z["shared_ff"], "shared_limit": LIMIT})


def _linear_spec(case):
    z = SHAPES[case["shape"]]
    return PartSpec("gated_linear_attention", {
        "hidden_size": z["width"], "heads": z["state_heads"], "dim": STATE_DIM, "value_dim": STATE_DIM, "tau": TAU, "eps": EPS,
        "decay_rank": z["rank"]})


def _part(category, spec, seed):
    part = build_part(category, spec)
    runtime = Runtime(DEVICE, torch.bfloat16)
    part.load(WeightSource(_Weights(part.tensor_decls(), seed).tensor, runtime))
    return part


# ------------------------------------------------------------------ what a program has in hand, and its call
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prefill", "float32"):
        model = _model(case, seed)
        held = _contexts(case["context"], case["requests"]) if kind == "decode" else [0] * case["requests"]
        new = [1] * case["requests"] if kind == "decode" else _lengths(case["tokens"], case["requests"])
        total = [h + n + 1 for h, n in zip(held, new)]
        runner = ModelRunner(model, num_pages=sum(-(-t // PAGE) for t in total), page_tokens=PAGE, max_requests=64, prefix_caching=False)
        sequences = [runner.new_sequence() for _ in held]
        for upto in range(PAGE, max(total) + PAGE, PAGE):          # pages taken in turn, as growing requests take them
            for seq, t in zip(sequences, total):
                if upto - PAGE < t and not runner.reserve(seq, min(upto, t)):
                    raise RuntimeError("the pool is too small for the case")
        if kind == "decode":
            heads, dim = QWEN_05B["num_key_value_heads"], 64
            width = max(len(seq.tables[0]) for seq in sequences)
            table = torch.tensor([list(seq.tables[0]) + [-1] * (width - len(seq.tables[0])) for seq in sequences], device=DEVICE)
            for slot in range(len(runner.storage.keys)):
                _place(runner.storage.keys[slot], table, _held_rows(seed, f"keys.{slot}", held, heads, dim))
                _place(runner.storage.values[slot], table, _held_rows(seed, f"values.{slot}", held, heads, dim))
        entries = [StepEntry(seq, tokens, [len(tokens) - 1]) for seq, tokens in zip(sequences, _tokens(seed, new))]
        return {"case": case, "runner": runner, "entries": entries, "held": held}
    z = SHAPES[case["shape"]]
    if kind == "experts":
        part = _part("feed_forward", _expert_spec(case), seed)
        return {"case": case, "part": part, "h": _normal(seed, "h", (case["tokens"], z["width"]), 1.0, torch.bfloat16)}
    if kind == "linear_attention":
        part = _part("mixer", _linear_spec(case), seed)
        new = _lengths(case["tokens"], case["requests"])
        ctx, _ = _step_context(new, [0] * len(new), seed)
        buffer = torch.zeros((len(new), *part.state_spec().shape), dtype=torch.float32, device=DEVICE)
        return {"case": case, "part": part, "ctx": ctx, "state": StateView(buffer, ctx.state_slots),
                "h": _normal(seed, "h", (case["tokens"], z["width"]), 1.0, torch.bfloat16)}
    part = _part("mixer", _map_spec(case) if kind == "map_attention" else _latent_spec(case), seed)
    new, held = _attention_case(case)
    ctx, pages = _step_context(new, held, seed)
    spec = part.cache_spec()
    keys = torch.zeros((pages, spec.kv_heads, PAGE, spec.head_dim), dtype=torch.bfloat16, device=DEVICE)
    values = torch.zeros((pages, spec.kv_heads, PAGE, spec.value_width), dtype=torch.bfloat16, device=DEVICE) if spec.value_width else None
    _place(keys, ctx.block_tables[0], _held_rows(seed, "keys", held, spec.kv_heads, spec.head_dim))
    if values is not None:
        _place(values, ctx.block_tables[0], _held_rows(seed, "values", held, spec.kv_heads, spec.value_width))
    return {"case": case, "part": part, "ctx": ctx, "cache": CacheView(keys, values, ctx.block_tables[0], PAGE, True),
            "h": _normal(seed, "h", (sum(new), z["width"]), 1.0, torch.bfloat16)}


def run(state):
    kind = state["case"]["kind"]
    if kind in ("decode", "prefill", "float32"):
        runner, entries = state["runner"], state["entries"]
        for entry, held in zip(entries, state["held"]):
            entry.seq.length = held
        if kind != "decode":
            return {"logits": runner.step(entries), "keys": runner.storage.keys, "values": runner.storage.values}
        none = [0.0] * len(entries)
        runner.step_and_sample(entries, none, none)
        return {"logits": runner.last_decode_graph.last_logits}
    h = state["h"]
    x = torch.zeros(h.shape, dtype=torch.float32, device=h.device)
    if kind == "experts":
        state["part"].forward(h, x)
        return {"x": x}
    if kind == "linear_attention":
        state["state"].buffer.zero_()                                # the requests are new
        state["part"].forward(h, x, state["ctx"], None, state["state"])
        return {"x": x, "state": state["state"].buffer}
    cache = state["cache"]
    state["part"].forward(h, x, state["ctx"], cache)
    return {"x": x, "keys": cache.k} if cache.v is None else {"x": x, "keys": cache.k, "values": cache.v}


# ------------------------------------------------------------------ what a pass cannot do without
def _visible(new, held, window=None):
    """(query, key) pairs that a causal mask, with a window or without, lets through."""
    pairs = 0
    for n, h in zip(new, held):
        if window is None:
            pairs += n * h + n * (n + 1) // 2
        else:
            pairs += sum(min(window, h + j + 1) for j in range(n))
    return pairs


def work(case):
    kind = case["kind"]
    if kind in ("decode", "prefill", "float32"):
        c = QWEN_05B
        layers, item = (4, 4) if kind == "float32" else (c["num_hidden_layers"], 2)
        hidden, ff, kv = c["hidden_size"], c["intermediate_size"], 2 * 64
        held = _contexts(case["context"], case["requests"]) if kind == "decode" else [0] * case["requests"]
        new = [1] * case["requests"] if kind == "decode" else _lengths(case["tokens"], case["requests"])
        matrices = layers * (hidden * (hidden + 2 * kv) + hidden * hidden + 3 * hidden * ff)
        head = hidden * c["vocab_size"]
        pairs = _visible(new, held)
        cache = layers * 2 * kv * item * (sum(held) + 2 * sum(new))
        return {"bytes": (matrices + head) * item + cache + 4 * c["vocab_size"] * case["requests"] + sum(new) * hidden * item,
                "flops": 2 * matrices * sum(new) + 2 * head * case["requests"] + layers * 4 * pairs * hidden}
    z = SHAPES[case["shape"]]
    width = z["width"]
    if kind == "experts":
        t = case["tokens"]
        outputs = z["experts"] + z["identity"]
        taken = t * TOP * z["experts"] / outputs                        # rows that go to an expert with weights
        unit, shared = 3 * width * z["expert_ff"], 3 * width * z["shared_ff"]
        reached = z["experts"] * (1.0 - (1.0 - TOP / outputs) ** t)
        return {"bytes": 2 * (reached * unit + shared) + 4 * outputs * width + t * width * (2 + 4 + 4),
                "flops": 2 * taken * unit + 2 * t * shared + 2 * t * outputs * width}
    if kind == "linear_attention":
        t, heads = case["tokens"], z["state_heads"]
        inner = heads * STATE_DIM
        weights = 4 * width * inner + z["rank"] * (width + inner) + inner * width
        return {"bytes": 2 * weights + t * width * (2 + 4 + 4) + 2 * 4 * case["requests"] * inner * STATE_DIM,
                "flops": 2 * weights * t + 4 * t * inner * STATE_DIM}
    new, held = _attention_case(case)
    tokens, rows = sum(new), sum(h + n for h, n in zip(held, new))
    if kind == "latent_attention":
        heads, rank = z["heads"], z["kv_rank"]
        weights = width * (z["q_rank"] + rank + 64) + z["q_rank"] * heads * 128 + heads * rank * (64 + 128) + heads * 128 * width
        # the arithmetic of the unfolded form, whose keys and values are made once per cached row
        return {"bytes": 2 * weights + tokens * width * (2 + 4 + 4) + 2 * (rank + 64) * (rows + tokens),
                "flops": 2 * weights * tokens + 2 * heads * rank * (64 + 128) * (rows - tokens) + 2 * _visible(new, held) * heads * (128 + 128)}
    q, k, v = z["heads"] * case["maps"] * case["dim"], z["kv_heads"] * case["maps"] * case["dim"], z["kv_heads"] * 128
    gates = z["heads"] if case["extras"] or case["mask"] == "window" else 0
    window = z["window"] if case["mask"] == "window" else None
    weights = width * (q + k + v + gates) + z["heads"] * 128 * width
    seen = sum(min(h, window) if window else h for h in held) + tokens
    return {"bytes": 2 * weights + tokens * width * (2 + 4 + 4) + 2 * (k + v) * (seen + tokens),
            "flops": 2 * weights * tokens + 2 * _visible(new, held, window) * z["heads"] * case["maps"] * (case["dim"] + 128)}


def tolerance(case):
    # four times the largest distance seen between the path and ``exact`` over seeds and drawn cases
    # (a decode step's split products add in any order: the same step twice differs by up to 0.015, 0.02 from ``exact``)
    return {"rel": {"decode": 0.07, "prefill": 0.03, "float32": 1e-5, "map_attention": 0.02, "latent_attention": 0.015,
                    "experts": 0.011, "linear_attention": 0.016}[case["kind"]]}


# ------------------------------------------------------------------ the same in float64
def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, positions, theta, dims, interleaved=False):
    """x [tokens, vectors, dim] with its first ``dims`` elements turned by the position."""
    frequency = theta ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    angle = positions.double()[:, None] * frequency
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]
    turned, rest = x[..., :dims], x[..., dims:]
    a, b = (turned[..., 0::2], turned[..., 1::2]) if interleaved else (turned[..., :dims // 2], turned[..., dims // 2:])
    first, second = a * cos - b * sin, b * cos + a * sin
    turned = torch.stack((first, second), -1).flatten(-2) if interleaved else torch.cat((first, second), -1)
    return torch.cat((turned, rest), -1)


def _softmax_attention(q, k, v, positions, scale, window=None, softcap=0.0, sink=None):
    """One head: q [new, dim] at ``positions`` over k, v of positions 0, 1, ...; [new, value_dim]."""
    score = (q @ k.T) * scale
    if softcap:
        score = softcap * torch.tanh(score / softcap)
    at = torch.arange(k.shape[0], device=q.device)
    hidden = at[None] > positions[:, None]
    if window is not None:
        hidden |= at[None] <= positions[:, None] - window
    score = score.masked_fill(hidden, -math.inf)
    top = score.max(-1, keepdim=True).values if sink is None else torch.clamp(score.max(-1, keepdim=True).values, min=float(sink))
    weight = torch.exp(score - top)
    total = weight.sum(-1, keepdim=True)
    if sink is not None:
        total = total + torch.exp(sink - top)
    return (weight @ v) / total


def _positions(new, held):
    return [torch.arange(h, h + n, device=DEVICE) for n, h in zip(new, held)]


def _exact_model(case, seed):
    c, w = QWEN_05B, _Exact(seed)
    layers = 4 if case["kind"] == "float32" else c["num_hidden_layers"]
    hidden, ff, heads, kv = c["hidden_size"], c["intermediate_size"], 14, 2
    decode = case["kind"] == "decode"
    held = _contexts(case["context"], case["requests"]) if decode else [0] * case["requests"]
    new = [1] * case["requests"] if decode else _lengths(case["tokens"], case["requests"])
    embedding = _weight(seed, "model.embed_tokens.weight", (c["vocab_size"], hidden), "matrix")
    tokens = torch.tensor(sum(_tokens(seed, new), []), device=DEVICE)
    x = embedding[tokens].double()
    positions = torch.cat(_positions(new, held))
    for layer in range(layers):
        p = f"model.layers.{layer}."
        h = _rms(x, c["rms_norm_eps"]) * w(p + "input_layernorm.weight", hidden, init="gain")

        def project(name, rows):
            return h @ w(f"{p}self_attn.{name}_proj.weight", rows, hidden).T + w(f"{p}self_attn.{name}_proj.bias", rows, init="bias")
        q = _rotate(project("q", heads * 64).reshape(-1, heads, 64), positions, c["rope_theta"], 64)
        k = _rotate(project("k", kv * 64).reshape(-1, kv, 64), positions, c["rope_theta"], 64)
        v = project("v", kv * 64).reshape(-1, kv, 64)
        k_held = _held_rows(seed, f"keys.{layer}", held, kv, 64) if decode else [k[:0]] * len(new)
        v_held = _held_rows(seed, f"values.{layer}", held, kv, 64) if decode else [v[:0]] * len(new)
        mixed, at = [], 0
        for i, n in enumerate(new):
            keys = torch.cat((k_held[i].double(), k[at:at + n]))
            values = torch.cat((v_held[i].double(), v[at:at + n]))
            mixed.append(torch.stack([_softmax_attention(q[at:at + n, j], keys[:, j // (heads // kv)], values[:, j // (heads // kv)],
                                                         positions[at:at + n], 0.125) for j in range(heads)], 1).flatten(1))
            at += n
        x = x + torch.cat(mixed) @ w(p + "self_attn.o_proj.weight", hidden, heads * 64).T
        h = _rms(x, c["rms_norm_eps"]) * w(p + "post_attention_layernorm.weight", hidden, init="gain")
        act = torch.nn.functional.silu(h @ w(p + "mlp.gate_proj.weight", ff, hidden).T) * (h @ w(p + "mlp.up_proj.weight", ff, hidden).T)
        x = x + act @ w(p + "mlp.down_proj.weight", hidden, ff).T
    last = torch.tensor(new, device=DEVICE).cumsum(0) - 1
    h = _rms(x[last], c["rms_norm_eps"]) * w("model.norm.weight", hidden, init="gain")
    # where a request's rows lie in the pool is the cache manager's choice
    return {"logits": h @ embedding.double().T} | ({} if decode else {"keys": [None] * layers, "values": [None] * layers})


def _exact_map_attention(case, seed):
    z, w = SHAPES[case["shape"]], _Exact(seed)
    width, heads, kv, maps, dim = z["width"], z["heads"], z["kv_heads"], case["maps"], case["dim"]
    new, held = _attention_case(case)
    ctx, pages = _step_context(new, held, seed)
    h = _normal(seed, "h", (sum(new), width), 1.0, torch.bfloat16).double()
    positions = torch.cat(_positions(new, held))
    q = _rotate((h @ w("q", heads * maps * dim, width).T).reshape(-1, heads * maps, dim), positions, 10000.0, 64)
    k = _rotate((h @ w("k", kv * maps * dim, width).T).reshape(-1, kv * maps, dim), positions, 10000.0, 64).reshape(-1, kv, maps * dim)
    v = (h @ w("v", kv * 128, width).T).reshape(-1, kv, 128)
    keys, values = torch.zeros((pages, kv, PAGE, maps * dim), dtype=torch.float64, device=DEVICE), \
        torch.zeros((pages, kv, PAGE, 128), dtype=torch.float64, device=DEVICE)
    k_held, v_held = _held_rows(seed, "keys", held, kv, maps * dim), _held_rows(seed, "values", held, kv, 128)
    k_all = [torch.cat((a.double(), b)) for a, b in zip(k_held, k.split(new))]
    v_all = [torch.cat((a.double(), b)) for a, b in zip(v_held, v.split(new))]
    _place(keys, ctx.block_tables[0], k_all)
    _place(values, ctx.block_tables[0], v_all)
    window = z["window"] if case["mask"] == "window" else None
    sink = w("sink", heads, init="bias") if case["extras"] else None
    lam = 0.0
    if maps == 2:
        lq1, lk1, lq2, lk2 = (w(name, dim, init="wide") for name in ("lq1", "lk1", "lq2", "lk2"))
        lam = torch.exp(lq1 @ lk1) - torch.exp(lq2 @ lk2) + 0.5
    mixed, at = [], 0
    for i, n in enumerate(new):
        where, out = positions[at:at + n], []
        for j in range(heads):
            g = j // (heads // kv)
            a = [_softmax_attention(q[at:at + n, j * maps + m], k_all[i][:, g, m * dim:(m + 1) * dim], v_all[i][:, g], where, dim ** -0.5,
                                    window, case["softcap"], None if sink is None else sink[j]) for m in range(maps)]
            out.append(a[0] if maps == 1 else _rms(a[0] - lam * a[1], EPS) * 0.5)
        mixed.append(torch.stack(out, 1))
        at += n
    mixed = torch.cat(mixed)
    if case["extras"] or window:
        mixed = mixed * torch.sigmoid(h @ w("g", heads, width).T)[..., None]
    return {"x": mixed.flatten(1) @ w("o", width, heads * 128).T, "keys": keys, "values": values}


def _exact_latent(case, seed):
    z, w = SHAPES[case["shape"]], _Exact(seed)
    width, heads, rank, q_rank = z["width"], z["heads"], z["kv_rank"], z["q_rank"]
    new, held = _attention_case(case)
    ctx, pages = _step_context(new, held, seed)
    h = _normal(seed, "h", (sum(new), width), 1.0, torch.bfloat16).double()
    positions = torch.cat(_positions(new, held))
    rows = h @ w("dkv", rank + 64, width).T
    c = _rms(rows[:, :rank], EPS) * w("dkv.norm", rank, init="gain")
    row = torch.cat((c, _rotate(rows[:, None, rank:], positions, 10000.0, 64, interleaved=True)[:, 0]), -1)
    q = _rms(h @ w("dq", q_rank, width).T, EPS) * w("dq.norm", q_rank, init="gain")
    q = (q @ w("uq", heads * 128, q_rank).T).reshape(-1, heads, 128)
    q = torch.cat((q[..., :64], _rotate(q[..., 64:], positions, 10000.0, 64, interleaved=True)), -1)
    uk, uv = w("uk", heads * 64, rank).reshape(heads, 64, rank), w("uv", heads * 128, rank).reshape(heads, 128, rank)
    sink = w("sink", heads, init="bias")
    rows_all = [torch.cat((a[:, 0].double(), b)) for a, b in zip(_held_rows(seed, "keys", held, 1, rank + 64), row.split(new))]
    keys = torch.zeros((pages, 1, PAGE, rank + 64), dtype=torch.float64, device=DEVICE)
    _place(keys, ctx.block_tables[0], [r[:, None] for r in rows_all])
    mixed, at = [], 0
    for i, n in enumerate(new):
        c_all, k_rot = rows_all[i][:, :rank], rows_all[i][:, rank:]
        mixed.append(torch.stack([_softmax_attention(q[at:at + n, j], torch.cat((c_all @ uk[j].T, k_rot), -1), c_all @ uv[j].T,
                                                     positions[at:at + n], 128 ** -0.5, sink=sink[j]) for j in range(heads)], 1))
        at += n
    return {"x": torch.cat(mixed).flatten(1) @ w("o", width, heads * 128).T, "keys": keys}


def _exact_experts(case, seed):
    z, w = SHAPES[case["shape"]], _Exact(seed)
    width, experts, identity = z["width"], z["experts"], z["identity"]
    h = _normal(seed, "h", (case["tokens"], width), 1.0, torch.bfloat16).double()

    def unit(rows, stem, ff):
        gate = torch.clamp(rows @ w(stem + "gate", ff, width).T, max=LIMIT)
        up = torch.clamp(rows @ w(stem + "up", ff, width).T, -LIMIT, LIMIT)
        return (gate * torch.sigmoid(ALPHA * gate) * (up + 1.0)) @ w(stem + "down", width, ff).T
    s = torch.softmax(h @ w("router", experts + identity, width, init="bias").T, -1)
    chosen = torch.topk(s + w("correction", experts + identity, init="bias"), TOP, dim=-1).indices
    weight = torch.gather(s, 1, chosen)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
    x = unit(h, "shared.", z["shared_ff"])
    for e in range(experts + identity):
        token, place = torch.nonzero(chosen == e, as_tuple=True)
        if token.numel():
            rows = h[token]
            x[token] += weight[token, place][:, None] * (unit(rows, f"e{e}.", z["expert_ff"]) if e < experts else rows)
    return {"x": x}


def _exact_linear_attention(case, seed):
    z, w = SHAPES[case["shape"]], _Exact(seed)
    width, heads = z["width"], z["state_heads"]
    inner = heads * STATE_DIM
    new = _lengths(case["tokens"], case["requests"])
    h = _normal(seed, "h", (case["tokens"], width), 1.0, torch.bfloat16).double()
    q, k, v = ((h @ w(name, inner, width).T).reshape(-1, heads, STATE_DIM) for name in ("q", "k", "v"))
    z_decay = (h @ w("a1", z["rank"], width).T) @ w("a2", inner, z["rank"]).T + w("a2.b", inner, init="bias")
    decay = torch.sigmoid(z_decay).pow(1.0 / TAU).reshape(-1, heads, STATE_DIM)
    # all requests' recurrences side by side, token by token; a request that has ended keeps its state
    state = torch.zeros((len(new), heads, STATE_DIM, STATE_DIM), dtype=torch.float64, device=DEVICE)
    out = torch.zeros_like(q)
    starts = [sum(new[:i]) for i in range(len(new))]
    for t in range(max(new)):
        live = [i for i, n in enumerate(new) if t < n]
        rows = torch.tensor([starts[i] + t for i in live], device=DEVICE)
        if len(live) == len(new):
            state = state * decay[rows][..., None] + k[rows][..., None] * v[rows][..., None, :]
            out[rows] = torch.einsum("rhdv,rhd->rhv", state, q[rows])
        else:
            which = torch.tensor(live, device=DEVICE)
            state[which] = state[which] * decay[rows][..., None] + k[rows][..., None] * v[rows][..., None, :]
            out[rows] = torch.einsum("rhdv,rhd->rhv", state[which], q[rows])
    out = _rms(out * STATE_DIM ** -0.5, EPS) * w("norm", STATE_DIM, init="gain")
    gate = torch.nn.functional.silu(h @ w("g", inner, width).T)
    return {"x": (out.flatten(1) * gate) @ w("o", width, inner).T, "state": state}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "prefill", "float32"):
        return _exact_model(case, seed)
    return {"map_attention": _exact_map_attention, "latent_attention": _exact_latent, "experts": _exact_experts,
            "linear_attention": _exact_linear_attention}[kind](case, seed)
