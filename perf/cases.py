"""What the engine is timed on: one step of a served model, from host token lists to logits on the device.

A case says a model, the run type and what the step holds: `decode` requests with one new token each behind `least` to
`context` cached ones, and `prompts` portions of `tokens` tokens behind `cached` ones (several: of half of that to all of
it).  Logits are wanted at the last place of every request, or at every place of the portions (`want` "all", as perplexity and replay
tools read them).

Models: the three Llama shapes that the engine is made for, and of its other designs the one with a latent cache, a
windowed cache and matrix memories.  The designs with a mixture of experts are not here: which experts a token
takes hangs on the last bit of a 16-bit input, so the results of two correct implementations cannot be held side by side.
"""

from __future__ import annotations

import hashlib
import math
import random
from typing import Dict, List

import torch

from bare_cuda_4gib_b200.engine.engine import LLMEngine
from bare_cuda_4gib_b200.engine.step import StepEntry
from bare_cuda_4gib_b200.models.presets import preset_config

F64 = torch.float64
STEP_TOKENS = 2048       # the engine's usual budget of prompt tokens a step
LLAMAS = ("tinyllama", "llama2-7b", "llama3-8b")
OTHERS = ("zadurax-2048",)
# The larger Llama shapes run 8 of their 32 layers: behind all of them, with weights of N(0, 0.02), 16-bit rounding alone
# moves the logits by 0.05 of their norm, and no two correct implementations could be told from wrong ones.
LAYERS = {"llama2-7b": 8, "llama3-8b": 8}


def _case(model, dtype="bfloat16", decode=0, least=0, context=0, prompts=0, tokens=0, cached=0, want="last"):
    return {"model": model, "dtype": dtype, "decode": decode, "least": least, "context": context, "prompts": prompts,
            "tokens": tokens, "cached": cached, "want": want}


def listed() -> List[dict]:
    return [
        # one person in a chat: the next token, where the time is the chain of launches and the weights
        dict(_case("tinyllama", decode=1, least=1000, context=1000), name="decode 1"),
        # the benchmark's steady decoding: eight requests at the end of the model's context
        dict(_case("tinyllama", decode=8, least=2047, context=2047), name="decode 8"),
        # a busy server: 64 requests, each somewhere else in its text
        dict(_case("tinyllama", decode=64, least=512, context=2047), name="decode 64 ragged"),
        # a question of a line: time to the first token
        dict(_case("tinyllama", prompts=1, tokens=61), name="prompt 61"),
        # the longest prompt the model takes, in one step
        dict(_case("tinyllama", prompts=1, tokens=2048), name="prompt 2048"),
        # continuous batching: decoding requests share the step with the prompts of new ones
        dict(_case("tinyllama", decode=24, least=100, context=1500, prompts=3, tokens=389), name="mixed 24 + 3"),
        # the larger models (8 layers): bound by their weights when decoding, by the tensor cores in a long prompt's second portion
        dict(_case("llama3-8b", decode=8, least=100, context=3001), name="8b decode 8"),
        dict(_case("llama2-7b", prompts=1, tokens=2048, cached=2048), name="7b prompt portion"),
        # the 32-bit run that answers are checked against: replayed token by token, and a window of a perplexity run
        dict(_case("tinyllama", "float32", decode=4, least=100, context=300), name="float32 decode 4"),
        dict(_case("tinyllama", "float32", prompts=1, tokens=257, want="all"), name="float32 window"),
        # a design with other mixers, both directions
        dict(_case("zadurax-2048", prompts=1, tokens=2048), name="zadurax prompt"),
        dict(_case("zadurax-2048", decode=8, least=700, context=1500), name="zadurax decode 8"),
    ]


def _spread(rng, low, high):
    """A whole number whose logarithm is uniform."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(("decode", "decode", "prompt", "prompt", "mixed"))
    model = rng.choice(("tinyllama",) * 4 + ("llama2-7b", "llama3-8b", "zadurax-2048"))
    big, other = model in ("llama2-7b", "llama3-8b"), model in OTHERS
    dtype = "float32" if model == "tinyllama" and rng.random() < 0.25 else "bfloat16"
    wide = dtype == "float32"
    if kind == "mixed" and other:
        kind = "decode"
    if kind == "decode":
        rows = _spread(rng, 1, 16 if wide or big else 64)
        context = _spread(rng, 16, 600 if wide else 2000)
        return _case(model, dtype, rows, max(1, int(context * rng.uniform(0.2, 1.0))), context)
    if kind == "prompt":
        tokens = _spread(rng, 1, 400 if wide else 1900)
        cached = rng.randrange(1, 2048 - tokens) if not (wide or other) and tokens < 1800 and rng.random() < 0.4 else 0
        return _case(model, dtype, prompts=1, tokens=tokens, cached=cached,
                     want="all" if tokens <= 600 and rng.random() < 0.25 else "last")
    rows = _spread(rng, 1, 8 if wide or big else 32)
    context = _spread(rng, 16, 400 if wide else 1800)
    return _case(model, dtype, rows, max(1, context // 3), context, prompts=rng.randrange(1, 4),
                 tokens=_spread(rng, 2, 100 if wide else 500))


# ----------------------------------------------------------------------------- the step

def _config(case):
    model = case["model"]
    return preset_config(model, num_hidden_layers=LAYERS[model]) if model in LAYERS else preset_config(model)


def _requests(case, seed):
    """(tokens in the cache before the step, tokens of the step) per request."""
    rng = random.Random(f"requests {seed}")
    vocab = _config(case).to_dict()
    vocab = vocab.get("vocab_size") or vocab["vocab"]
    lengths = [(rng.randint(case["least"], case["context"]), 1) for _ in range(case["decode"])]
    lengths += [(case["cached"], rng.randint(max(1, case["tokens"] // 2), case["tokens"]) if case["prompts"] > 1 else case["tokens"])
                for _ in range(case["prompts"])]
    return [([rng.randrange(vocab) for _ in range(a)], [rng.randrange(vocab) for _ in range(b)]) for a, b in lengths]


def _wanted(case, at, n):
    return list(range(n)) if case["want"] == "all" and at >= case["decode"] else [n - 1]


def prepare(case, seed):
    """The loaded engine, the requests' earlier tokens in its cache, and the next step's entries."""
    requests = _requests(case, seed)
    config, longest = _config(case), max(case["context"] + 1, case["cached"] + case["tokens"])
    engine = LLMEngine(None, max_tokens=longest, max_seqs=len(requests), dtype=case["dtype"], page_tokens=64,
                       max_step_tokens=STEP_TOKENS + len(requests), random=(config, seed))
    slots = []
    for before, _new in requests:
        slot = engine.cache.acquire_slot()
        for at in range(0, len(before), STEP_TOKENS):
            engine.runner.step([StepEntry(slot, before[at: at + STEP_TOKENS])])
        slots.append(slot)
    return {"engine": engine, "slots": slots, "fresh": [not before for before, _ in requests],
            "tokens": [new for _, new in requests], "wanted": [_wanted(case, i, len(new)) for i, (_, new) in enumerate(requests)]}


def run(state):
    """One step; afterwards every request goes back to where it was, as it does where several continuations of one
    text are tried (matrix memories run on), and a prompt that began in this step takes a slot anew and gives it back."""
    engine, slots = state["engine"], list(state["slots"])
    cache, runner = engine.cache, engine.runner
    for i, fresh in enumerate(state["fresh"]):
        if fresh:
            cache.release_slot(slots[i])
    for i, fresh in enumerate(state["fresh"]):
        if fresh:
            slots[i] = cache.acquire_slot()
    state["slots"] = slots
    logits = runner.step([StepEntry(s, t, w) for s, t, w in zip(slots, state["tokens"], state["wanted"])])
    for slot, tokens, fresh in zip(slots, state["tokens"], state["fresh"]):
        if not fresh:
            cache.commit(slot, -len(tokens))
    return {"logits": logits, "cached": [g.storage for g in cache.groups], "memories": [m for _, m in sorted(cache.states.items())]}


# ----------------------------------------------------------------------------- what a pass cannot do without

def _sizes(case):
    """(weights in the layers and the head, vocabulary, width, layer runs, per layer run (score and value multiplications
    per query and key, cached numbers per position, window))."""
    d = _config(case).to_dict()
    if case["model"] in LLAMAS:
        width, heads, ff, vocab, layers = (d["hidden_size"], d["num_attention_heads"], d["intermediate_size"], d["vocab_size"],
                                           d["num_hidden_layers"])
        kv, dim = d["num_key_value_heads"], d.get("head_dim") or d["hidden_size"] // d["num_attention_heads"]
        own = (heads + 2 * kv) * dim * width + heads * dim * width + 3 * width * ff
        return own * layers + vocab * width, own * layers, vocab, width, [(2 * heads * dim, 2 * kv * dim, None, 0)] * layers
    width, vocab = d["width"], d["vocab"]
    stored = multiplied = 0
    mixers = []
    for layer in d["layers"]:
        m, ff = layer["mixer"], layer["mlp"]["ff"]
        H, dim = m["heads"], m["dim"]
        if layer["type"] == "attention":
            own = width * dim * (2 * H + m["kv_heads"]) + H * dim * width
            mixers.append((2 * H * dim, 2 * m["kv_heads"] * dim, m["mask"]["size"], 0))
        elif layer["type"] == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            own = width * (H * (dim + m["rot_dim"]) + row + H * m["vdim"]) + H * (dim + m["vdim"]) * m["kv_rank"] + H * m["vdim"] * width
            mixers.append((H * (dim + m["rot_dim"] + m["vdim"]), row, None, 0))
        else:
            own = width * H * (2 * dim + 2 * m["vdim"] + 2) + H * m["vdim"] * width
            mixers.append((0, 0, None, H * dim * (m["vdim"] + 1)))
        own += 3 * width * ff
        multiplied += own
        if "weights_of" not in layer:
            stored += own
    return stored + vocab * width, multiplied, vocab, width, mixers


def work(case) -> Dict[str, float]:
    stored, multiplied, vocab, width, mixers = _sizes(case)
    size = 4 if case["dtype"] == "float32" else 2
    requests = [(len(a), len(b)) for a, b in _requests(case, 0)]
    tokens = sum(n for _, n in requests)
    wanted = sum(len(_wanted(case, i, n)) for i, (_, n) in enumerate(requests))
    nbytes = stored * size + tokens * width * size + wanted * vocab * 4
    flops = 2.0 * multiplied * tokens + 2.0 * wanted * vocab * width
    for products, row, window, memory in mixers:
        for before, n in requests:
            seen = before if window is None else min(before, window - 1)
            nbytes += (seen + n) * row * size + 8 * memory
            pairs = sum(min(before + i + 1, window or before + i + 1) for i in range(n))
            flops += 2.0 * products * pairs + 6.0 * memory * n
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # against `exact` the float32 logits measured 2.6e-6 to 3.3e-6 and the bfloat16 ones 0.009 to 0.02 (22 layers whose
    # inputs are rounded to 8 bits at every product)
    if case["dtype"] == "float32":
        return {"rel": 1.3e-5}
    return {"rel": 0.03, "max": 0.6}


# ----------------------------------------------------------------------------- the same in 64 bits

def _tensor(seed, name, shape, kind="matrix"):
    """The seeded weights, as the engine's random mode states them: a generator per tensor from the seed and the
    tensor's name, 0.02 N(0, 1) for matrices, 1 + 0.01 N(0, 1) for norms, N(0, 1) for "unit", rounded to bfloat16."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int.from_bytes(hashlib.sha256(f"{seed}:{name}".encode()).digest()[:8], "little") & 0x7FFFFFFFFFFFFFFF)
    x = torch.randn(shape, generator=g, dtype=torch.float32, device="cuda")
    x = 1.0 + 0.01 * x if kind == "norm" else x if kind == "unit" else 0.02 * x
    return x.to(torch.bfloat16).to(F64)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _softmax_values(q, k, v, scale, before, window=None, sink=None):
    """q [n, H, d] at positions before.., k [m, G, d], v [m, G, e], head h reading group h // (H / G): [n, H, e]."""
    n, H = q.shape[:2]
    m, G = k.shape[:2]
    j = torch.arange(m, device=q.device)
    out = torch.empty(n, H, v.shape[-1], dtype=F64, device=q.device)
    for at in range(0, n, 1024):
        rows = q[at: at + 1024]
        i = before + at + torch.arange(rows.shape[0], device=q.device)[:, None]
        hidden = j[None] > i if window is None else (j[None] > i) | (i - j[None] >= window)
        s = torch.einsum("ighd,jgd->ghij", rows.view(rows.shape[0], G, H // G, -1), k) * scale
        s.masked_fill_(hidden, -math.inf)
        if sink is None:
            p = torch.softmax(s, -1)
        else:
            extra = sink.view(G, H // G, 1, 1)
            top = torch.maximum(s.amax(-1, keepdim=True), extra)
            p = torch.exp(s - top)
            p = p / (p.sum(-1, keepdim=True) + torch.exp(extra - top))
        out[at: at + 1024] = torch.einsum("ghij,jge->ighe", p, v).reshape(rows.shape[0], H, -1)
    return out


def _exact_llama(d, seed, requests, wanted):
    width, heads, kv, eps = d["hidden_size"], d["num_attention_heads"], d["num_key_value_heads"], d["rms_norm_eps"]
    dim, ff = d.get("head_dim") or width // heads, d["intermediate_size"]
    lengths = [len(t) for t in requests]
    ids = torch.tensor([i for t in requests for i in t], device="cuda")
    place = torch.cat([torch.arange(n, device="cuda") for n in lengths]).to(F64)
    # the inverse frequencies are a table of 32-bit numbers
    freq = 1.0 / d["rope_theta"] ** (torch.arange(dim // 2, dtype=torch.float32) * 2 / dim)
    angle = place[:, None] * freq.to(F64).cuda()[None]
    cos, sin = torch.cos(angle)[:, None], torch.sin(angle)[:, None]

    def turned(x):
        a, b = x[..., : dim // 2], x[..., dim // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = _tensor(seed, "model.embed_tokens.weight", (d["vocab_size"], width))[ids]
    for i in range(d["num_hidden_layers"]):
        p = f"model.layers.{i}."

        def product(h, name, rows, cols):
            return h @ _tensor(seed, f"{p}{name}.weight", (rows, cols)).T

        h = _rms(x, eps) * _tensor(seed, p + "input_layernorm.weight", (width,), "norm")
        q = turned(product(h, "self_attn.q_proj", heads * dim, width).view(-1, heads, dim))
        k = turned(product(h, "self_attn.k_proj", kv * dim, width).view(-1, kv, dim))
        v = product(h, "self_attn.v_proj", kv * dim, width).view(-1, kv, dim)
        o = torch.cat([_softmax_values(a, b, c, dim ** -0.5, 0)
                       for a, b, c in zip(q.split(lengths), k.split(lengths), v.split(lengths))])
        x = x + product(o.reshape(-1, heads * dim), "self_attn.o_proj", width, heads * dim)
        h = _rms(x, eps) * _tensor(seed, p + "post_attention_layernorm.weight", (width,), "norm")
        gate, up = product(h, "mlp.gate_proj", ff, width), product(h, "mlp.up_proj", ff, width)
        x = x + product(torch.nn.functional.silu(gate) * up, "mlp.down_proj", width, ff)
    x = _rms(x[wanted], eps) * _tensor(seed, "model.norm.weight", (width,), "norm")
    head = "model.embed_tokens.weight" if d.get("tie_word_embeddings") else "lm_head.weight"
    return x @ _tensor(seed, head, (d["vocab_size"], width)).T


def _turned_pairs(x, place, rot):
    """x [n, heads, d]: of the first `dims` entries, 2i and 2i + 1 turned by place * base^(-2i / dims); with `scaling`
    slow pairs turn `factor` times slower, by a ramp over the pairs, and cos and sin grow."""
    dims, base, scaling = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    freq, grown = base ** (-2.0 * i / dims), 1.0
    if scaling:
        low, high = (dims * math.log(scaling["original"] / (2 * math.pi * scaling[k])) / (2 * math.log(base)) for k in ("fast", "slow"))
        low, high = max(math.floor(low), 0), min(math.ceil(high), dims - 1)
        ramp = ((i - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        freq, grown = freq / scaling["factor"] * ramp + freq * (1.0 - ramp), 0.1 * math.log(scaling["factor"]) + 1.0
    angle = place[:, None] * freq[None]
    cos, sin = (torch.cos(angle) * grown)[:, None], (torch.sin(angle) * grown)[:, None]
    out = x.clone()
    out[..., 0:dims:2] = x[..., 0:dims:2] * cos - x[..., 1:dims:2] * sin
    out[..., 1:dims:2] = x[..., 1:dims:2] * cos + x[..., 0:dims:2] * sin
    return out


def _matrix_memory(q, k, v, write, keep):
    """q, k [n, H, d], v [n, H, e], log gates [n, H]: the memory S_t = keep S + write k v^T read by q, over
    max(|n.q|, 1) in the scale of the largest log gate, all pairs at once."""
    F = torch.cumsum(keep, 0).T                                            # [H, n]
    w = F[:, :, None] - F[:, None, :] + write.T[:, None, :]
    w = w.masked_fill(torch.ones(w.shape[1:], dtype=torch.bool, device=w.device).triu(1), -math.inf)
    top = torch.maximum(w.amax(-1), F)
    a = torch.exp(w - top[..., None]) * torch.einsum("ihd,jhd->hij", q, k)
    below = torch.maximum(a.sum(-1).abs(), torch.exp(-top)) + 1e-6
    return (torch.einsum("hij,jhe->hie", a, v) / below[..., None]).transpose(0, 1)


def _exact_zadurax(d, seed, tokens, wanted):
    width, eps, n = d["width"], d["norm"]["eps"], len(tokens)
    place = torch.arange(n, device="cuda", dtype=F64)

    def norm(x, name, size=width):
        return _rms(x, eps) * _tensor(seed, name, (size,), "norm")

    x = norm(_tensor(seed, "embed", (d["vocab"], width))[torch.tensor(tokens, device="cuda")], "embed.norm")
    for i, layer in enumerate(d["layers"]):
        p, m = f"l{layer.get('weights_of', i)}.", layer["mixer"]
        H, dim = m["heads"], m["dim"]

        def product(h, name, rows):
            return h @ _tensor(seed, p + name, (rows, h.shape[-1])).T

        h = norm(x, p + "norm1")
        if layer["type"] == "attention":
            G = m["kv_heads"]
            q, k = product(h, "mix.q", H * dim).view(n, H, dim), product(h, "mix.k", G * dim).view(n, G, dim)
            o = _softmax_values(_turned_pairs(norm(q, p + "mix.q.norm", dim), place, m["rot"]),
                                _turned_pairs(norm(k, p + "mix.k.norm", dim), place, m["rot"]), k, m["scale"], 0, m["mask"]["size"])
        elif layer["type"] == "latent_attention":
            rot, rank, e = m["rot_dim"], m["kv_rank"], m["vdim"]
            q = product(h, "mix.q", H * (dim + rot)).view(n, H, dim + rot)
            down = product(h, "mix.dkv", rank + rot)
            latent = norm(down[:, :rank], p + "mix.dkv.norm", rank)
            key = torch.cat([product(latent, "mix.uk", H * dim).view(n, H, dim),
                             _turned_pairs(down[:, None, rank:], place, m["rot"]).expand(n, H, rot)], -1)
            o = _softmax_values(torch.cat([q[..., :dim], _turned_pairs(q[..., dim:], place, m["rot"])], -1), key,
                                product(latent, "mix.uv", H * e).view(n, H, e), m["scale"], 0,
                                sink=_tensor(seed, p + "mix.sink", (H,), "unit"))
        else:
            e, cap = m["vdim"], m["gate_cap"]
            q, k = product(h, "mix.q", H * dim).view(n, H, dim) * dim ** -0.5, product(h, "mix.k", H * dim).view(n, H, dim)
            v = product(h, "mix.v", H * e).view(n, H, e)
            write, keep = (cap * torch.tanh((product(h, f"mix.{g}", H) + _tensor(seed, f"{p}mix.{g}.b", (H,), "unit")) / cap) for g in "if")
            o = _rms(_matrix_memory(q, k, v, write, torch.nn.functional.logsigmoid(keep)), eps)
            o = o.reshape(n, H * e) * _tensor(seed, p + "mix.norm", (H * e,), "norm")
        o = o.reshape(n, -1)
        o = o * torch.sigmoid(product(h, "mix.g", o.shape[-1]))
        x = x + norm(product(o, "mix.o", width), p + "norm1b")
        h = norm(x, p + "norm2")
        ff = layer["mlp"]["ff"]
        gate, up = product(h, "mlp.gate", ff), product(h, "mlp.up", ff)
        x = x + norm(product(torch.nn.functional.gelu(gate, approximate="tanh") * up, "mlp.down", width), p + "norm2b")
    return norm(x[wanted], "final.norm") @ _tensor(seed, "head", (d["vocab"], width)).T


def exact(case, seed):
    """Logits of the step in 64 bits, every request's text from its first token on."""
    requests = _requests(case, seed)
    d = _config(case).to_dict()
    texts = [a + b for a, b in requests]
    if case["model"] in LLAMAS:
        wanted, start = [], 0
        for i, (before, new) in enumerate(requests):
            wanted += [start + len(before) + w for w in _wanted(case, i, len(new))]
            start += len(before) + len(new)
        logits = _exact_llama(d, seed, texts, torch.tensor(wanted, device="cuda"))
    else:
        logits = torch.cat([_exact_zadurax(d, seed, text, torch.tensor([len(before) + w for w in _wanted(case, i, len(new))], device="cuda"))
                            for i, (text, (before, new)) in enumerate(zip(texts, requests))])
    return {"logits": logits, "cached": None, "memories": None}
