"""The work that this library is timed on: steps of `Engine.step` and draws of `BatchSampler`, with
random weights of the sizes that `llm_b200.shapes` and the tests know.

A step case says which model runs (`model`, `layers` of it, `dtype`), how many sequences the step
has (`batch`), how many tokens each of them already holds in the cache (`held_low` to `held_high`,
spread evenly over the batch), how many new tokens each brings (`new_low` to `new_high`) and whether
the logits of every new token are wanted or those of each sequence's last one (`all_logits`). A step
with no held tokens is a prefill, one with one new token a sequence a decode step, anything else a
prompt that goes on (the next turn of a conversation). A `sample` case draws one token for every row
of a step's logits with the command line's parameters.

Large models run with some of their layers (8 of the Llama shapes' 32, 4 of the other architectures',
the head with its full vocabulary); the sizes of the layers are the shapes' own.
"""
from __future__ import annotations

import math
import zlib

import torch

from llm_b200.config import config_from_dict
from llm_b200.engine import DecoderModel, Engine, Entry
from llm_b200.sampling import BatchSampler, SamplingParams
from llm_b200.shapes import shape

DEVICE = "cuda:0"
BACK = ("o_proj.weight", "down_proj.weight", ".o", ".down")      # the matrices that lead back into the stream
DECODED_BEFORE = 3                 # tokens that a decoding sequence has already been given one by one

# the small configuration of the 32-bit runs (a model folder of the tests)
TINY = {
    "architectures": ["LlamaForCausalLM"], "model_type": "llama", "num_hidden_layers": 2, "hidden_size": 64,
    "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 16, "intermediate_size": 172, "vocab_size": 256,
    "rope_theta": 10000.0, "rope_scaling": None, "rms_norm_eps": 1e-5, "tie_word_embeddings": True,
    "attention_bias": False, "max_position_embeddings": 128, "hidden_act": "silu", "eos_token_id": 2,
}


# ----------------------------------------------------------------------------- the cases

def _step(name, model, layers, batch, held, new, dtype="bfloat16", all_logits=False):
    return {"name": name, "kind": "step", "model": model, "layers": layers, "dtype": dtype, "batch": batch,
            "held_low": held[0], "held_high": held[1], "new_low": new[0], "new_high": new[1], "all_logits": all_logits}


def listed():
    return [
        # the smallest call: a step of the 32-bit path on a small model, three unequal sequences (logit comparison runs)
        _step("tiny_decode_fp32", "tiny", 2, 3, (5, 17), (1, 1), dtype="float32"),
        # one user, a short conversation: the latency of a token
        _step("llama8b_decode_1", "llama-3.1-8b", 8, 1, (512, 512), (1, 1)),
        # the benchmark's headline: eight long contexts
        _step("llama8b_decode_8", "llama-3.1-8b", 8, 8, (7900, 8100), (1, 1)),
        # many unequal sequences on the whole of a small model
        _step("llama1b_decode_64", "llama-3.2-1b", 16, 64, (1, 8190), (1, 1)),
        # one prompt, the benchmark's prefill
        _step("llama8b_prefill_2048", "llama-3.1-8b", 8, 1, (0, 0), (2048, 2048)),
        # the next turn of two conversations: short odd prompts behind what the cache holds
        _step("llama8b_next_turn", "llama-3.1-8b", 8, 2, (700, 1501), (93, 257)),
        # many unequal prompts at once, one key head per query head
        _step("llama7b_prefill_16", "llama-2-7b", 8, 16, (0, 0), (64, 2048)),
        # the other mixers and feed-forwards: differential attention
        _step("guberax_prefill", "guberax-8b", 4, 1, (0, 0), (3001, 3001)),
        # delta rule, windowed attention and routed experts: two prompts, and a batch that decodes
        _step("zogapel_prefill", "zogapel-8b", 4, 2, (0, 0), (777, 1300)),
        _step("zogapel_decode_24", "zogapel-8b", 4, 24, (100, 2500), (1, 1)),
        # latent attention, mixed sigmoid attention and a gated recurrence
        _step("mefolorn_prefill", "mefolorn-8b", 4, 1, (0, 0), (2500, 2500)),
        # the draw behind a decode step of 32 sequences
        {"name": "sample_32", "kind": "sample", "batch": 32, "vocab": 128256, "temperature": 0.7},
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.randrange(11)
    if kind == 0:
        low = rng.randint(1, 30)
        case = _step("", "tiny", 2, rng.randint(1, 8), (low, low + rng.randint(0, 60)), (1, 1), dtype="float32")
    elif kind in (1, 2):
        low = _log(rng, 64, 7000)
        case = _step("", "llama-3.1-8b", 8, _log(rng, 1, 8), (low, low + rng.randint(0, 1100)), (1, 1))
    elif kind == 3:
        case = _step("", "llama-3.2-1b", 16, _log(rng, 9, 64), (1, _log(rng, 200, 8190)), (1, 1))
    elif kind == 4:
        n = _log(rng, 16, 2048)
        case = _step("", "llama-3.1-8b", 8, 1, (0, 0), (n, n))
    elif kind == 5:
        low, held = _log(rng, 16, 300), _log(rng, 64, 2000)
        case = _step("", "llama-3.1-8b", 8, rng.randint(1, 4), (held, held + rng.randint(0, 1000)), (low, low + rng.randint(0, 200)))
    elif kind == 6:
        case = _step("", "llama-2-7b", 8, _log(rng, 2, 16), (0, 0), (rng.randint(32, 200), _log(rng, 300, 2048)))
    elif kind == 7:
        n = _log(rng, 64, 4096)
        case = _step("", "guberax-8b", 4, 1, (0, 0), (n, n))
    elif kind == 8:
        low = _log(rng, 32, 1000)
        case = _step("", "zogapel-8b", 4, rng.randint(1, 4), (0, 0), (low, low + rng.randint(0, 800)))
    elif kind == 9:
        low = _log(rng, 64, 1000)
        case = _step("", "zogapel-8b", 4, _log(rng, 1, 64), (low, low + rng.randint(0, 1500)), (1, 1))
    else:
        n = _log(rng, 64, 3000)
        case = _step("", "mefolorn-8b", 4, 1, (0, 0), (n, n))
    if rng.random() < 0.08:
        case = {"kind": "sample", "batch": _log(rng, 1, 64), "vocab": rng.choice((32000, 128256)), "temperature": rng.choice((0.6, 0.7, 0.9))}
    case.pop("name", None)
    return case


# ----------------------------------------------------------------------------- inputs

def _raw(case):
    """The config.json contents of the case's model."""
    return dict(TINY) if case["model"] == "tiny" else shape(case["model"], case["layers"])


def _spread(batch, low, high):
    """`batch` whole numbers from low to high, evenly spread, long and short ones mixed."""
    at = [low + (high - low) * i // max(batch - 1, 1) for i in range(batch)]
    stride = next(s for s in (7, 5, 3, 1) if math.gcd(s, batch) == 1)
    return [at[i * stride % batch] for i in range(batch)]


def _lengths(case):
    """Per sequence, the tokens it holds before the step and those it brings."""
    return (_spread(case["batch"], case["held_low"], case["held_high"]),
            _spread(case["batch"], case["new_low"], case["new_high"]))


def _tokens(case, seed, vocab):
    """Per sequence, the ids of the held and the new tokens."""
    gen = torch.Generator().manual_seed(seed * 7919 + 17)
    return [(torch.randint(0, vocab, (h,), generator=gen).tolist(), torch.randint(0, vocab, (n,), generator=gen).tolist())
            for h, n in zip(*_lengths(case))]


def _weight(name, spec, seed, dtype):
    """One random tensor by its name: matrices N(0, 0.02), gains around one (or around zero where they are stored as an
    offset), taps of the order of 1 / taps. As in a trained model, a layer changes the stream by a part of its size
    (embedding rows of unit size, the matrices that lead back into the stream a quarter as large), and a router's
    choices are decided (its rows three times as large)."""
    gen = torch.Generator(device=DEVICE).manual_seed((seed * 0x9E3779B1 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFFFFFF)
    t = torch.empty(spec.shape, dtype=dtype, device=DEVICE).normal_(generator=gen)
    if spec.role == "gain":
        return t.mul_(0.02).add_(1.0)
    if spec.role == "gate_scalar":
        return t.mul_(0.02).add_(0.5)
    if spec.role == "taps":
        return t.mul_(1.0 / spec.shape[-1])
    if "embed" in name:
        return t
    return t.mul_(0.06 if name.endswith("router") else 0.005 if name.endswith(BACK) else 0.02)


def _weights(case, model, seed):
    dtype = getattr(torch, case["dtype"])
    return {name: _weight(name, spec, seed, dtype) for name, spec in model.parameters().items()}


def prepare(case, seed):
    if case["kind"] == "sample":
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        logits = torch.empty((case["batch"], case["vocab"]), device=DEVICE).normal_(generator=gen).mul_(1.3)
        params = [SamplingParams(temperature=case["temperature"], seed=seed * 1000 + i) for i in range(case["batch"])]
        return {"sampler": BatchSampler(params, case["vocab"], DEVICE), "next": logits, "logits": torch.empty_like(logits),
                "rows": list(range(case["batch"]))}
    config = config_from_dict(_raw(case))
    model = DecoderModel(config.model_spec())
    model.bind(_weights(case, model, seed), getattr(torch, case["dtype"]), DEVICE)
    held, new = _lengths(case)
    context = max(h + n for h, n in zip(held, new))
    engine = Engine(model, max_tokens=sum((h + n + 63) // 64 * 64 for h, n in zip(held, new)), max_seq_len=context,
                    max_slots=case["batch"])
    tokens = _tokens(case, seed, model.spec.vocab)
    wants = [list(range(len(n))) if case["all_logits"] else [len(n) - 1] for _, n in tokens]
    if not any(held):                                           # prompts: the slots are taken by the call
        return {"engine": engine, "slots": None, "held": held, "tokens": tokens, "wants": wants}
    slots = engine.acquire(case["batch"])
    given = [min(DECODED_BEFORE, h - 1) if max(new) == 1 else 0 for h in held]
    engine.step([Entry(s, h[:len(h) - g], []) for s, (h, _), g in zip(slots, tokens, given)])
    for k in range(DECODED_BEFORE):
        entries = [Entry(s, [h[len(h) - g + k]], [0]) for s, (h, _), g in zip(slots, tokens, given) if k < g]
        if entries:
            engine.step(entries)
    return {"engine": engine, "slots": slots, "held": held, "tokens": tokens, "wants": wants}


# ----------------------------------------------------------------------------- one pass

def run(state):
    if "sampler" in state:
        state["logits"].copy_(state["next"])                    # a step's logits: the sampler's chain writes into them
        return state["sampler"].sample(state["logits"], state["rows"])
    engine = state["engine"]
    slots = state["slots"] or engine.acquire(len(state["tokens"]))
    logits = engine.step([Entry(s, n, w) for s, (_, n), w in zip(slots, state["tokens"], state["wants"])])
    if state["slots"] is None:
        engine.release(slots)
    else:                                                       # back to the place before the step
        for s, h in zip(slots, state["held"]):
            engine.cache.set_length(s, h)
    # what the step wrote: keys and values, and the states of layers that keep one
    cache = [t for g in engine.cache.groups for t in ((g.storage,) if g.storage is not None else (g.keys, g.values))]
    return {"logits": logits, "cache": cache, "state": [t for t in engine.cache.states if t is not None]}


# ----------------------------------------------------------------------------- what a pass cannot do without

def _attended(held, new, window):
    """Query-key pairs of a step, and the distinct keys it reads."""
    pairs = keys = 0
    for h, n in zip(held, new):
        if window and h + n > window:
            pairs += sum(min(p + 1, window) for p in range(h, h + n))
            keys += min(h + n, window + n)
        else:
            pairs += n * h + n * (n + 1) // 2
            keys += h + n
    return pairs, keys


def work(case):
    if case["kind"] == "sample":
        n = case["batch"] * case["vocab"]
        return {"bytes": 4.0 * n + 4.0 * case["batch"], "flops": 4.0 * n}
    raw = _raw(case)
    spec = config_from_dict(raw).model_spec()
    model = DecoderModel(spec)
    held, new = _lengths(case)
    tokens = sum(new)
    rows = tokens if case["all_logits"] else case["batch"]
    size = 4 if case["dtype"] == "float32" else 2
    head = spec.vocab * spec.hidden
    nbytes, flops = float(size * head + 4 * rows * spec.vocab + size * tokens * spec.hidden), 2.0 * rows * head
    for name, p in model.parameters().items():
        count = math.prod(p.shape)
        if name in (spec.embedding, spec.head) or len(p.shape) < 2:
            continue
        used, share = 1.0, 1.0
        if ".mlp.e" in name:                                    # one of the routed experts
            router = next(l["mlp"]["router"] for l in raw["layers"] if l["mlp"].get("router"))
            share = router["top"] / router["experts"]
            used = 1.0 - (1.0 - share) ** tokens
        nbytes += size * count * used
        flops += 2.0 * tokens * count * share
    for kv, layer in zip(DecoderModel(spec).cache_requests()[0], raw.get("layers") or [None] * len(spec.schedule)):
        m = (layer or {}).get("mixer") or {}
        m = m.get("left") or m
        if kv is not None:
            pairs, keys = _attended(held, new, (m.get("mask") or {}).get("size", 0))
            heads = m.get("heads") or raw["num_attention_heads"]
            key, value = kv.head_dim, getattr(kv, "value_dim", None) or kv.head_dim
            one = kv.n_kv_heads * (key + (value if (layer or {}).get("type") != "latent_attention" else 0))
            nbytes += size * (keys + tokens) * one
            flops += 2.0 * pairs * heads * (key + value) * (1.5 if case["model"].startswith("guberax") else 1.0)
        if (layer or {}).get("type") == "delta":
            states = m["heads"] * m["dim"] * m["vdim"]
            nbytes += 4.0 * states * case["batch"] * (2 if any(held) else 1)
            flops += 6.0 * tokens * states
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "sample":
        return "exact"
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-4}
    # bfloat16: measured against the unfolded norms and another kernel for the products, 0.004 to 0.008 (Llama, Guberax)
    # and 0.012 (Zogapel, where a token whose last expert is a near tie differs in single values); 64 bits are 0.004 to
    # 0.006 away from Llama and Guberax, 0.013 from Mefolorn, 0.017 to 0.020 from Zogapel
    if case["model"].startswith("zogapel"):
        return {"rel": 0.03, "max": 0.95}
    return {"rel": 0.03 if case["model"].startswith("mefolorn") else 0.02, "max": 0.3}


# ----------------------------------------------------------------------------- the same in 64 bits

F = torch.float64


class _Doubles:
    """The case's weights in 64 bits, made when they are asked for."""

    def __init__(self, case, seed):
        self.specs = DecoderModel(config_from_dict(_raw(case)).model_spec()).parameters()
        self.seed, self.dtype = seed, getattr(torch, case["dtype"])

    def __getitem__(self, name):
        return _weight(name, self.specs[name], self.seed, self.dtype).to(F)


def _rms(x, gain, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _frequencies(dims, base, scaling):
    """One frequency per rotated pair, and the factor of cosine and sine."""
    freq = base ** (-2.0 * torch.arange(dims // 2, dtype=F) / dims)
    if not scaling:
        return freq.to(DEVICE), 1.0
    factor = float(scaling["factor"])
    if "fast" in scaling:                                       # a ramp over the pairs, with a larger magnitude
        def dim_of(turns):
            return dims * math.log(scaling["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        low, high = max(math.floor(dim_of(scaling["fast"])), 0), min(math.ceil(dim_of(scaling["slow"])), dims - 1)
        ramp = ((torch.arange(dims // 2, dtype=F) - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
        return (freq / factor * ramp + freq * (1.0 - ramp)).to(DEVICE), 0.1 * math.log(factor) + 1.0
    low = scaling.get("low_freq_factor", scaling.get("low"))
    high = scaling.get("high_freq_factor", scaling.get("high"))
    original = scaling.get("original_max_position_embeddings", scaling.get("original"))
    blend = ((original * freq / (2.0 * math.pi) - low) / (high - low)).clamp(0.0, 1.0)
    return ((1.0 - blend) * freq / factor + blend * freq).to(DEVICE), 1.0


def _rotate(x, dims, base, scaling, pairs="half"):
    """x [T, heads, dim] of a whole sequence: the first `dims` elements of every head turn."""
    freq, magnitude = _frequencies(dims, float(base), scaling)
    angle = torch.arange(x.shape[0], dtype=F, device=DEVICE)[:, None, None] * freq
    c, s = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude
    out = x.clone()
    one, two = (slice(0, dims, 2), slice(1, dims, 2)) if pairs == "next" else (slice(0, dims // 2), slice(dims // 2, dims))
    out[..., one] = x[..., one] * c - x[..., two] * s
    out[..., two] = x[..., two] * c + x[..., one] * s
    return out


def _seen(n, window):
    i = torch.arange(n, device=DEVICE)
    seen = i[None, :] <= i[:, None]
    return seen & (i[:, None] - i[None, :] < window) if window else seen


def _attend(q, k, v, scale, window=0, sink=None):
    """One head's softmax attention over a whole sequence, with the sink's term in the denominator."""
    s = (q @ k.T).mul_(scale).masked_fill_(~_seen(q.shape[0], window), -math.inf)
    if sink is None:
        return torch.softmax(s, -1) @ v
    top = torch.maximum(s.amax(-1, keepdim=True), sink)
    e = torch.exp(s - top)
    return (e / (e.sum(-1, keepdim=True) + torch.exp(sink - top))) @ v


def _conv(u, taps, bias=0.0):
    padded = torch.cat([torch.zeros(taps.shape[1] - 1, u.shape[1], dtype=F, device=DEVICE), u])
    return bias + sum(taps[:, j] * padded[j:j + u.shape[0]] for j in range(taps.shape[1]))


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _gated(h, w):
    return (_silu(h @ w("gate").T) * (h @ w("up").T)) @ w("down").T


def _llama_layer(raw, x, seqs, w, i):
    p, eps = f"model.layers.{i}.", raw["rms_norm_eps"]
    heads, groups, dim = raw["num_attention_heads"], raw["num_key_value_heads"], raw["head_dim"]
    wq, wk, wv, wo = (w[p + f"self_attn.{r}_proj.weight"] for r in "qkvo")
    gate, up, down = (w[p + f"mlp.{r}_proj.weight"] for r in ("gate", "up", "down"))
    n1, n2 = w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"]
    for a, b in seqs:
        h = _rms(x[a:b], n1, eps)
        q, k = (_rotate((h @ m.T).view(b - a, -1, dim), dim, raw["rope_theta"], raw["rope_scaling"]) for m in (wq, wk))
        v = (h @ wv.T).view(b - a, groups, dim)
        o = [_attend(q[:, e], k[:, e * groups // heads], v[:, e * groups // heads], dim ** -0.5) for e in range(heads)]
        x[a:b] += torch.cat(o, -1) @ wo.T
        h = _rms(x[a:b], n2, eps)
        x[a:b] += (_silu(h @ gate.T) * (h @ up.T)) @ down.T


def _guberax_layer(raw, x, seqs, w, i):
    p, m, eps = f"l{i}.", raw["layers"][i]["mixer"], raw["norm"]["eps"]
    heads, groups, dim, rot = m["heads"], m["kv_heads"], m["dim"], m["rot"]
    mix = {n: w[p + "mix." + n] for n in ("q", "k", "v", "o", "q.conv", "k.conv", "v.conv", "lq1", "lk1", "lq2", "lk2")}
    lam = torch.exp((mix["lq1"] * mix["lk1"]).sum()) - torch.exp((mix["lq2"] * mix["lk2"]).sum()) + m["diff"]
    for a, b in seqs:
        h = _rms(x[a:b], 1.0 + w[p + "norm1"], eps)
        q, k, v = (_conv(h @ mix[r].T, mix[r + ".conv"]) for r in "qkv")
        q, k = (_rotate(t.view(b - a, -1, dim), rot["dims"], rot["base"], rot["scaling"], "next") for t in (q, k))
        v = v.view(b - a, groups, m["vdim"])
        out = []
        for e in range(heads):
            g = e * groups // heads
            d = _attend(q[:, 2 * e], k[:, 2 * g], v[:, g], m["scale"]) - lam * _attend(q[:, 2 * e + 1], k[:, 2 * g + 1], v[:, g], m["scale"])
            out.append(_rms(d, 1.0 - m["diff"], eps))
        x[a:b] += torch.cat(out, -1) @ mix["o"].T + _gated(h, lambda n: w[p + "mlp." + n])


def _delta(h, m, w, eps):
    heads, groups, dim, vdim = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (_silu(_conv(h @ w(r).T, w(r + ".conv"))).view(h.shape[0], -1, d) for r, d in (("q", dim), ("k", dim), ("v", vdim)))
    q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(heads // groups, 1) for t in (q * dim ** -0.5, k))
    beta = torch.sigmoid(h @ w("b").T)
    decay = torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(h @ w("a").T + w("dt_bias")))
    state, out = torch.zeros(heads, dim, vdim, dtype=F, device=DEVICE), torch.empty_like(v)
    for t in range(h.shape[0]):
        state *= decay[t, :, None, None]
        u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None], state)[:, 0])
        torch.baddbmm(state, k[t, :, :, None], u[:, None], out=state)
        out[t] = torch.bmm(q[t, :, None], state)[:, 0]
    out = _rms(out, w("norm"), eps) * _silu(h @ w("g").T).view_as(out)
    return out.reshape(h.shape[0], -1) @ w("o").T


def _zogapel_attention(h, m, w):
    heads, groups, dim, n = m["heads"], m["kv_heads"], m["dim"], h.shape[0]
    q, v = (h @ w("q").T).view(n, heads, dim), (h @ w("k").T).view(n, groups, dim)
    q, k = (_rotate(t, m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]) for t in (q, v))
    o = [_attend(q[:, e], k[:, e * groups // heads], v[:, e * groups // heads], m["scale"], m["mask"]["size"]) for e in range(heads)]
    return (torch.cat(o, -1) * torch.sigmoid(h @ w("g").T)) @ w("o").T


def _experts(h, f, w):
    logits = h @ w("router").T + w("router.b")
    best = torch.topk(logits, f["router"]["top"], -1)
    share = torch.zeros_like(logits).scatter_(1, best.indices, torch.softmax(best.values, -1))
    out = torch.zeros_like(h)
    for e in range(f["router"]["experts"]):
        at = share[:, e].nonzero()[:, 0]
        out[at] += share[at, e, None] * _gated(h[at], lambda n: w(f"e{e}.{n}"))
    return out


def _zogapel_layer(raw, x, seqs, w, i):
    p, layer, eps = f"l{i}.", raw["layers"][i], raw["norm"]["eps"]
    held = {}

    def mix(name):
        return held.setdefault(name, w[p + "mix." + name])
    for a, b in seqs:
        h = _rms(x[a:b], 1.0 + w[p + "norm1"], eps)
        y = _delta(h, layer["mixer"], mix, eps) if layer["type"] == "delta" else _zogapel_attention(h, layer["mixer"], mix)
        x[a:b] += _rms(y, 1.0 + w[p + "norm1b"], eps)
    held.clear()
    for a in range(0, x.shape[0], 16384):
        h = _rms(x[a:a + 16384], 1.0 + w[p + "norm2"], eps)
        if layer["mlp"]["kind"] == "dense":
            y = _gelu(h @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T
        else:
            y = _experts(h, layer["mlp"], lambda n: w[p + "mlp." + n])
        x[a:a + 16384] += _rms(y, 1.0 + w[p + "norm2b"], eps)


def _latent(h, m, w, eps):
    heads, n = m["heads"], h.shape[0]
    q = (_rms(h @ w("dq").T, w("dq.norm"), eps) @ w("uq").T).view(n, heads, m["dim"])
    c = _rms(h @ w("dkv").T, w("dkv.norm"), eps)
    k, v = (c @ w("uk").T).view(n, heads, m["dim"]), (c @ w("uv").T).view(n, heads, m["vdim"])
    sink, gate = w("sink"), torch.sigmoid(h @ w("g").T)
    o = [_attend(q[:, e], k[:, e], v[:, e], m["scale"], m["mask"]["size"], sink[e]) * gate[:, e:e + 1] for e in range(heads)]
    return torch.cat(o, -1) @ w("o").T


def _mixed_sigmoid(h, m, w, eps):
    heads, groups, dim, n = m["heads"], m["kv_heads"], m["dim"], h.shape[0]
    q, k = (_rms(h @ w(r).T, w(r + ".norm"), eps).view(n, -1, dim) for r in "qk")
    q, k = (_rotate(t, m["rot"]["dims"], m["rot"]["base"], None) for t in (q, k))
    v, out, talk = (h @ w("v").T).view(n, groups, m["vdim"]), torch.empty(n, heads, m["vdim"], dtype=F, device=DEVICE), w("talk")
    seen, k = _seen(n, m["mask"]["size"]), k.repeat_interleave(heads // groups, 1)
    for a in range(0, n, 512):                                  # all heads' scores of some queries
        s = torch.einsum("ihd,jhd->hij", q[a:a + 512], k) * m["scale"]
        s = torch.sigmoid(torch.einsum("hg,gij->hij", talk, s) + w("pb")[:, None, None]) * seen[a:a + 512]
        for e in range(heads):
            out[a:a + 512, e] = s[e] @ v[:, e * groups // heads]
    return out.reshape(n, -1) @ w("o").T


def _recurrence(h, m, w):
    y = _gelu(h @ w("y").T + w("y.b"))
    u = _conv(h @ w("x").T + w("x.b"), w("conv"), w("conv.b"))
    parts = u.view(u.shape[0], m["blocks"], -1)
    r, i = (torch.sigmoid(torch.einsum("tbi,boi->tbo", parts, w(g)) + w(g + ".b")).reshape(u.shape) for g in ("ra", "ri"))
    a = torch.exp(-8.0 * r * torch.nn.functional.softplus(w("lam")))
    drive = torch.sqrt(1.0 - a * a) * i * u
    state, out = torch.zeros_like(u[0]), torch.empty_like(u)
    for t in range(u.shape[0]):
        state = torch.addcmul(drive[t], a[t], state)
        out[t] = state
    return (out * y) @ w("o").T


def _mefolorn_layer(raw, x, seqs, w, i):
    p, layer, eps = f"l{i}.", raw["layers"][i], raw["norm"]["eps"]
    m = layer["mixer"]

    def norm(z, name):
        return torch.tanh(w[p + name + ".alpha"] * z) * w[p + name] + w[p + name + ".b"]
    for a, b in seqs:
        h = norm(x[a:b], "norm1")
        if layer["type"] == "latent_attention":
            y = _latent(h, m, lambda n: w[p + "mix." + n], eps)
        else:
            y = (m["left_scale"] * _mixed_sigmoid(h, m["left"], lambda n: w[p + "mix.left." + n], eps)
                 + m["right_scale"] * _recurrence(h, m["right"], lambda n: w[p + "mix.right." + n]))
        x[a:b] += y + _gated(norm(x[a:b], "norm2"), lambda n: w[p + "mlp." + n])


def exact(case, seed):
    logits = None if case["kind"] == "sample" else _logits(case, seed)      # (a sample is whole numbers only)
    return None if logits is None else {"logits": logits, "cache": None, "state": None}


def _logits(case, seed):
    raw, w = _raw(case), _Doubles(case, seed)
    family = "llama" if "num_hidden_layers" in raw else raw["architecture"].lower()
    layer = {"llama": _llama_layer, "guberax": _guberax_layer, "zogapel": _zogapel_layer, "mefolorn": _mefolorn_layer}[family]
    held, new = _lengths(case)
    vocab = raw.get("vocab_size") or raw["vocab"]
    ids, seqs, rows = [], [], []
    for (h, n), first in zip(_tokens(case, seed, vocab), range(case["batch"])):
        seqs.append((len(ids), len(ids) + len(h) + len(n)))
        ids += h + n
        rows += list(range(len(ids) - len(n) if case["all_logits"] else len(ids) - 1, len(ids)))
    embedding = w["model.embed_tokens.weight" if family == "llama" else "embed"]
    x = embedding[torch.tensor(ids, device=DEVICE)]
    for i in range(case["layers"]):
        layer(raw, x, seqs, w, i)
    x = x[rows]
    if family == "llama":
        return _rms(x, w["model.norm.weight"], raw["rms_norm_eps"]) @ (embedding if raw["tie_word_embeddings"] else w["lm_head.weight"]).T
    if family == "mefolorn":
        return (torch.tanh(w["final.norm.alpha"] * x) * w["final.norm"] + w["final.norm.b"]) @ embedding.T
    z = _rms(x, 1.0 + w["final.norm"], raw["norm"]["eps"])
    if family == "guberax":
        return raw["logit_softcap"] * torch.tanh(z @ w["head"].T / raw["logit_softcap"])
    return z @ embedding.T
