"""What this framework is used for, as cases that can be timed and compared.

Four kinds of work, all through the public entry points:

* ``linear``: one BitLinear layer on device rows (``TernaryLinear.forward_device``);
* ``ffn``: one gated feed-forward on device rows (``GatedFFN.forward_device``);
* ``prompt`` / ``steps`` / ``chat`` / ``generate``: the ternary model.  A prompt for its last logits, one token per
  sequence behind a filled cache, a prompt followed by such steps (what sampling with a temperature does), and
  device-resident greedy generation;
* ``likerax`` / ``miborax``: the two layer-described bf16 decoders, prompts and steps.

Everything is made on the GPU from the case and a seed.  ``exact`` restates each path in float64 from the same
weights; it shares no code with the product.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rotor-rag_b200"))

VOCAB = 128256
#: The two shapes of the ternary model this repository is built around (rotor_b200/synth.py).
SHAPES = {"2b": dict(d_model=2560, n_heads=20, n_kv_heads=5, d_ff=6912),
          "xl": dict(d_model=8192, n_heads=64, n_kv_heads=8, d_ff=28672)}
#: Likerax at the sizes of the first shape; Miborax as its benchmark has it.
LIKERAX = dict(vocab=VOCAB, d=2560, heads=20, kv=5, dim=128, ff=6912, streams=2, chunk=1024)
MIBORAX = dict(vocab=102400, d=2048, heads=16, dim=128, rot=64, vdim=128, rank=512, q_rank=1536, window=1024, experts=64, top=6,
               ff=1408)
EPS = {1: 1e-5, 3: 1e-6}
THETA = 500000.0


def listed():
    return [
        # one projection of the 2B model on one token: the product a plug-in asks for per call, the smallest use
        dict(name="linear_one_row", kind="linear", rows=1, inn=2560, out=6912, terms=1),
        # the same layer class at sizes that are multiples of nothing, a handful of rows, float-faithful activations
        # (three int8 terms, the constructor's default)
        dict(name="linear_ragged", kind="linear", rows=13, inn=1923, out=3001, terms=3),
        # the feed-forward block of the 2B model on a small batch
        dict(name="ffn_16_rows", kind="ffn", rows=16, d=2560, ff=6912, terms=1),
        # a short answer to a short prompt at the whole 2B shape: the latency a single user sees
        dict(name="generate_2b", kind="generate", shape="2b", layers=30, terms=1, batch=1, context=128, steps=32),
        # a small serving batch: one token for each of eight sequences
        dict(name="steps_2b_batch_8", kind="steps", shape="2b", layers=30, terms=1, batch=8, context=517, steps=4),
        # reading long prompts: a full context for eight sequences
        dict(name="prompt_2b_8x2048", kind="prompt", shape="2b", layers=30, terms=1, batch=8, context=2048, steps=0),
        # what the loader gives by default (the reference's float semantics): a prompt, then tokens drawn one by one
        dict(name="chat_2b_float", kind="chat", shape="2b", layers=30, terms=3, batch=1, context=301, steps=12),
        # a full serving batch of the large shape behind long contexts (four of its eighty layers)
        dict(name="steps_xl_batch_64", kind="steps", shape="xl", layers=4, terms=1, batch=64, context=1024, steps=2),
        # prompts of the hyper-connection decoder with chunked attention
        dict(name="likerax_prompt", kind="likerax", layers=6, batch=8, context=2048, steps=0),
        # a small serving batch of the latent-attention mixture of experts
        dict(name="miborax_steps", kind="miborax", layers=6, batch=8, context=1024, steps=4),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["linear", "linear", "ffn", "generate", "steps", "steps", "prompt", "chat", "likerax", "miborax"])
    terms = rng.choice([1, 1, 3])
    if kind == "linear":
        return dict(kind=kind, rows=log(1, 4096), inn=log(256, 8192), out=log(256, 8192), terms=terms)
    if kind == "ffn":
        d, ff = rng.choice([(2560, 6912), (1024, 2736), (4096, 11008)])
        return dict(kind=kind, rows=log(1, 2048), d=d, ff=ff, terms=terms)
    if kind in ("likerax", "miborax"):
        if rng.random() < 0.5:
            batch = rng.randint(1, 8)
            return dict(kind=kind, layers=6, batch=batch, context=log(20, 2048), steps=0)
        return dict(kind=kind, layers=6, batch=rng.randint(1, 16), context=log(64, 2000), steps=rng.randint(2, 6))
    if kind == "steps":
        shape = rng.choice(["2b", "2b", "xl"])
        layers = rng.randint(12, 30) if shape == "2b" else rng.randint(2, 4)
        return dict(kind=kind, shape=shape, layers=layers, terms=terms, batch=log(1, 64), context=log(64, 2000), steps=rng.randint(1, 4))
    layers = rng.randint(12, 30)
    if kind == "prompt":
        return dict(kind=kind, shape="2b", layers=layers, terms=1, batch=rng.randint(1, 8), context=log(64, 2048), steps=0)
    if kind == "chat":
        return dict(kind=kind, shape="2b", layers=layers, terms=terms, batch=rng.randint(1, 2), context=log(16, 700),
                    steps=rng.randint(4, 16))
    return dict(kind=kind, shape="2b", layers=layers, terms=1, batch=rng.randint(1, 8), context=log(8, 700), steps=rng.randint(8, 48))


# ------------------------------------------------------------------ seeded inputs, shared by prepare() and exact()
def generator(*key):
    g = torch.Generator(device="cuda")
    g.manual_seed(hash(tuple(int(k) for k in key)) & 0x7fffffffffff)
    return g


def ternary(g, out, inn):
    return torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8)


def ternary_layer(case, seed, i):
    """(matrices by name with their scales, sub-norm weights) of layer i.  The sub-norm gains are those of a network in which
    a layer moves the residual by a part of its size; the greedy choice then rests on margins as clear as a trained model's."""
    s = SHAPES[case["shape"]]
    d, ff, hd = s["d_model"], s["d_ff"], s["d_model"] // s["n_heads"]
    dkv = s["n_kv_heads"] * hd
    g, host = generator(seed, 1, i), np.random.default_rng([seed, i])
    sizes = dict(q=(d, d), k=(dkv, d), v=(dkv, d), o=(d, d), gate=(ff, d), up=(ff, d), down=(d, ff))
    mats = {n: (ternary(g, *shape), float(np.float32(0.8165 * shape[1] ** -0.5 * (1 + 0.25 * host.random())))) for n, shape in sizes.items()}
    norms = {n: (gain * (1 + 0.1 * host.standard_normal(k))).astype(np.float32)
             for n, k, gain in (("input", d, 1.0), ("post", d, 1.0), ("attn", d, 0.08), ("ffn", ff, 0.08))}
    return mats, norms


def ternary_embedding(case, seed):
    d = SHAPES[case["shape"]]["d_model"]
    return torch.randn((VOCAB, d), generator=generator(seed, 2), device="cuda", dtype=torch.float32).to(torch.bfloat16)


def cached_rows(case, seed, i):
    """What layer i has cached of the context: keys and values [batch, KV heads, context, head size]."""
    s = SHAPES[case["shape"]]
    g, hd = generator(seed, 3, i), s["d_model"] // s["n_heads"]
    shape = (case["batch"], s["n_kv_heads"], case["context"], hd)
    return [torch.randn(shape, generator=g, device="cuda") for _ in range(2)]


def tokens(case, seed, vocab):
    """(prompt or None, one row of tokens per step)."""
    host = np.random.default_rng([seed, 77])
    prompt = host.integers(0, vocab, size=(case["batch"], case["context"]))
    return prompt, host.integers(0, vocab, size=(case["steps"], case["batch"], 1))


def dense(g, out, inn):
    return (torch.randn((out, inn), generator=g, device="cuda") * inn ** -0.5).to(torch.bfloat16)


def likerax_layer(seed, i):
    c, g = LIKERAX, generator(seed, 4, i)
    d, n = c["d"], c["streams"]
    qd, kd = c["heads"] * c["dim"], c["kv"] * c["dim"]
    w = {k: dense(g, *shape) for k, shape in dict(q=(qd, d), k=(kd, d), v=(kd, d), o=(d, qd), gate=(c["ff"], d), up=(c["ff"], d),
                                                  down=(d, c["ff"])).items()}
    host = np.random.default_rng([seed, 4, i])
    for q in (1, 2):
        w[f"norm{q}"] = torch.tensor(1 + 0.1 * host.standard_normal(d), dtype=torch.float32)
        w[f"in{q}"] = torch.tensor(0.5 + 0.1 * host.standard_normal(n), dtype=torch.float32)
        w[f"out{q}"] = torch.tensor(1 + 0.2 * host.standard_normal(n), dtype=torch.float32)
        w[f"mix{q}"] = torch.tensor(0.9 * np.eye(n) + 0.05 * host.standard_normal((n, n)), dtype=torch.float32)
    return w


def miborax_layer(seed, i):
    """A windowed layer, one that reads its cache, and a layer over the whole past, in turn.  The first columns of the residual
    hold well separated values that no layer overwrites and the routers read, so that routing never hangs on a rounding."""
    c, g = MIBORAX, generator(seed, 5, i)
    d, h, ff, n, rank, rot = c["d"], c["heads"], c["ff"], c["experts"], c["rank"], c["rot"]
    full, lent = i % 3 == 2, i % 3 == 1
    rows = h * (c["dim"] + rot)

    def closed(m):
        m[:n] = 0
        return m

    w = dict(uk=dense(g, h * c["dim"], rank), uv=dense(g, h * c["vdim"], rank), o=closed(dense(g, d, h * c["vdim"])))
    if full:
        w.update(dq=dense(g, c["q_rank"], d), uq=dense(g, rows, c["q_rank"]), gate=dense(g, h, d))
    else:
        w["q"] = dense(g, rows, d)
    if not lent:
        w["dkv"] = dense(g, rank + rot, d)
    w["experts"] = [(dense(g, ff, d), dense(g, ff, d), closed(dense(g, d, ff))) for _ in range(n)]
    w["router"] = torch.eye(n, d, device="cuda", dtype=torch.bfloat16)
    w["sink"] = torch.randn(h, generator=g, device="cuda")
    return w, full, lent


def miborax_embedding(seed):
    c, g = MIBORAX, generator(seed, 6)
    e = torch.randn((c["vocab"], c["d"]), generator=g, device="cuda")
    place = torch.rand((c["vocab"], c["experts"]), generator=g, device="cuda").argsort(1)
    e[:, :c["experts"]] = torch.linspace(-1.7, 1.7, c["experts"], device="cuda")[place]
    return (e * c["d"] ** -0.5).to(torch.bfloat16)


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("linear", "ffn"):
        return dict(case=case, layer=layer_of(case, seed), x=rows_of(case, seed))
    if kind in ("likerax", "miborax"):
        return decoder_state(case, seed)
    from rotor_b200.synth import BitNetModel
    from rotor_b200.transformer import KVCache
    shape, total = SHAPES[case["shape"]], case["context"] + case["steps"]
    rows = case["batch"] * (1 if kind == "steps" else case["context"])
    capacity = max(total, 2048) if kind in ("generate", "chat") else total   # (2048: what the loader allocates when it is not told)
    model = BitNetModel(dict(shape, vocab_size=VOCAB, n_layers=case["layers"]), semantics=semantics_of(case), max_seq=capacity,
                        max_batch=case["batch"], max_rows=rows)
    model.embed_tokens = ternary_embedding(case, seed)
    for i, layer in enumerate(model.layers):
        mats, norms = ternary_layer(case, seed, i)
        a, f = layer.attention, layer.ffn
        for name, proj in dict(q=a.q_proj, k=a.k_proj, v=a.v_proj, o=a.o_proj, gate=f.gate_proj, up=f.up_proj, down=f.down_proj).items():
            proj.load_from_int8(*mats[name])
        layer.input_norm.weight, layer.post_attn_norm.weight = norms["input"], norms["post"]
        a.attn_norm.weight, f.ffn_norm.weight = norms["attn"], norms["ffn"]
    prompt, steps = tokens(case, seed, VOCAB)
    state = dict(case=case, model=model, prompt=prompt, steps=steps)
    if kind == "steps":
        for i, layer in enumerate(model.layers):
            for cache, rows in zip(layer.attention.ensure_cache(case["batch"], total), cached_rows(case, seed, i)):
                cache[:, :, :case["context"]] = rows
        state["caches"] = [KVCache(layer.attention, case["context"], case["batch"]) for layer in model.layers]
    return state


def semantics_of(case):
    from rotor_b200.semantics import BASELINE, REFERENCE
    return BASELINE if case["terms"] == 1 else REFERENCE


def layer_weights(case, seed):
    g, host = generator(seed, 7), np.random.default_rng([seed, 7])
    sizes = [(case["out"], case["inn"])] if case["kind"] == "linear" else [(case["ff"], case["d"])] * 2 + [(case["d"], case["ff"])]
    return [(ternary(g, *s), float(np.float32(s[1] ** -0.5 * (1 + 0.25 * host.random())))) for s in sizes]


def layer_of(case, seed):
    from rotor_b200.transformer import GatedFFN, TernaryLinear
    w = layer_weights(case, seed)
    if case["kind"] == "linear":
        layer = TernaryLinear(case["inn"], case["out"], semantics=semantics_of(case))
        layer.load_from_int8(*w[0])
        return layer
    layer = GatedFFN(case["d"], case["ff"], semantics=semantics_of(case))
    for proj, m in zip((layer.gate_proj, layer.up_proj, layer.down_proj), w):
        proj.load_from_int8(*m)
    return layer


def rows_of(case, seed):
    return torch.randn((case["rows"], case["inn"] if case["kind"] == "linear" else case["d"]), generator=generator(seed, 8), device="cuda")


def decoder_state(case, seed):
    from rotor_b200.decoder_model import Connections, DecoderModel, Experts, Latent, LayerSpec
    from rotor_b200.likerax import distance_slopes
    b, context = case["batch"], case["context"]
    sizes = dict(max_seq=context + case["steps"], max_batch=b, max_rows=b * context)
    specs = []
    if case["kind"] == "likerax":
        c = LIKERAX
        for i in range(case["layers"]):
            w = likerax_layer(seed, i)
            specs.append(LayerSpec(c["heads"], c["kv"], c["dim"], c["dim"], c["dim"] ** -0.5, w["q"], w["k"], w["v"], w["o"], w["norm1"],
                                   unit_qk=True, chunk=c["chunk"], slopes=distance_slopes(c["heads"]), gate=w["gate"], up=w["up"],
                                   down=w["down"], norm2=w["norm2"], hc1=Connections(w["in1"], w["out1"], w["mix1"]),
                                   hc2=Connections(w["in2"], w["out2"], w["mix2"])))
        g = generator(seed, 6)
        embed, head = dense(g, c["vocab"], c["d"]) * c["d"] ** 0.5, dense(g, c["vocab"], c["d"])
        model = DecoderModel(specs, list(range(case["layers"])), embed, head, torch.ones(c["d"]), streams=c["streams"], eps=1e-5, **sizes)
    else:
        c = MIBORAX
        one, zero = torch.ones(c["d"]), torch.zeros(c["d"])
        for i in range(case["layers"]):
            w, full, lent = miborax_layer(seed, i)
            a = Latent(c["rank"], c["rot"], 10000.0, w["uk"], w["uv"], kv_from=i - 1 if lent else None)
            if not lent:
                a.dkv, a.kv_norm = w["dkv"], torch.ones(c["rank"])
            if full:
                a.dq, a.q_norm, a.uq, a.gate = w["dq"], torch.ones(c["q_rank"]), w["uq"], w["gate"]
            gate, up, down = zip(*w["experts"])
            specs.append(LayerSpec(c["heads"], 1, c["dim"], c["vdim"], (c["dim"] + c["rot"]) ** -0.5, w.get("q"), None, None, w["o"], one,
                                   window=0 if full else c["window"], sinks=w["sink"], act="silu", norm1_b=zero, norm2=one, norm2_b=zero,
                                   parallel=True, latent=a, experts=Experts(c["top"], w["router"], gate, up, down, bias=torch.zeros(c["experts"]))))
        model = DecoderModel(specs, range(case["layers"]), miborax_embedding(seed), None, one, final_norm_b=zero, eps=1e-5,
                             embed_scale=c["d"] ** 0.5, **sizes)
    prompt, steps = tokens(case, seed, c["vocab"])
    state = dict(case=case, model=model, prompt=prompt, steps=steps)
    if case["steps"]:
        state["caches"] = model.forward_last_logits_device(prompt)[1]
    return state


# ------------------------------------------------------------------ run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("linear", "ffn"):
        return state["layer"].forward_device(state["x"])
    model = state["model"]
    if kind == "generate":
        from rotor_b200.transformer import KVCache
        new = model.generate_greedy_batch(state["prompt"], case["steps"])
        # the logits behind the last token, as a program that goes on from here would ask for them
        caches = [KVCache(layer.attention, case["context"] + case["steps"] - 1, case["batch"]) for layer in model.layers]
        return new, model.forward_last_logits_device(new[:, -1:], caches)[0]
    out, caches = [], state.get("caches")
    if caches is None:
        logits, caches = model.forward_last_logits_device(state["prompt"])
        out.append(logits)
    for ids in state["steps"]:
        logits, caches = model.forward_last_logits_device(ids, caches)
        out.append(logits)
    return out


# ------------------------------------------------------------------ work and tolerance
def visible_pairs(first, last, reach):
    """Query-key pairs of the positions first .. last - 1; reach: keys a query sees at most (0: all up to its own)."""
    return sum(min(i + 1, reach) if reach else i + 1 for i in range(first, last))


def work(case):
    kind = case["kind"]
    if kind in ("linear", "ffn"):
        inn, out, n = (case["inn"], case["out"], 1) if kind == "linear" else (case["d"], case["ff"], 3)
        ends = inn + out if kind == "linear" else 2 * inn
        return {"bytes": n * inn * out / 4 + 4.0 * case["rows"] * ends, "flops": 2.0 * n * inn * out * case["rows"]}
    b, context, steps, layers = case["batch"], case["context"], case["steps"], case["layers"]
    calls = steps + (1 if kind == "generate" else 0) + (0 if kind in ("steps", "generate") else 1)
    if kind in ("likerax", "miborax"):
        calls = steps if steps else 1
        rows = b * (steps if steps else context)
        first, last = (context, context + steps) if steps else (0, context)
        if kind == "likerax":
            c = LIKERAX
            per = (2 * c["heads"] + 2 * c["kv"]) * c["dim"] * c["d"] + 3 * c["ff"] * c["d"]
            held, row_bytes, heads, width = per, 2 * 2 * c["kv"] * c["dim"], c["heads"], 2 * c["dim"]
            pairs = layers * sum(i % c["chunk"] + 1 for i in range(first, last))
        else:
            c = MIBORAX
            expert = 3 * c["ff"] * c["d"]
            attention = c["heads"] * (c["dim"] + c["rot"]) * c["d"] + c["heads"] * (c["dim"] + c["vdim"]) * c["rank"] + \
                c["heads"] * c["vdim"] * c["d"] + (c["rank"] + c["rot"]) * c["d"]
            per = attention + c["top"] * expert
            rows_a_call = rows // calls
            met = c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** rows_a_call)  # experts that a call's tokens meet
            held = attention + met * expert
            row_bytes, heads, width = 2 * (c["rank"] + c["rot"]), c["heads"], c["dim"] + c["rot"] + c["vdim"]
            pairs = sum(visible_pairs(first, last, 0 if i % 3 == 2 else c["window"]) for i in range(layers))
        table = 2.0 * c["vocab"] * c["d"]
        read = layers * 2.0 * held + table
        kv = row_bytes * b * (pairs if steps else layers * context)
        head = 2.0 * calls * b * c["vocab"] * c["d"]
        return {"bytes": calls * read + kv + 4.0 * calls * b * c["vocab"],
                "flops": 2.0 * layers * per * rows + 2.0 * b * heads * width * pairs + head}
    s = SHAPES[case["shape"]]
    d, ff, dkv = s["d_model"], s["d_ff"], s["n_kv_heads"] * (s["d_model"] // s["n_heads"])
    per = 2 * d * d + 2 * d * dkv + 3 * d * ff
    prompt = 0 if kind == "steps" else context
    passes = calls if kind != "generate" else steps + 1     # the prompt, then one pass per further token and one for the logits
    rows = b * (prompt + passes - (1 if prompt else 0))
    first, last = context - prompt, context + passes - (1 if prompt else 0)
    pairs = layers * visible_pairs(context, last, 0) + layers * (visible_pairs(0, prompt, 0) if case["terms"] == 1 else prompt * prompt)
    weights = layers * per / 4 + 2.0 * VOCAB * d
    kv = 8.0 * dkv * b * (layers * visible_pairs(context, last, 0) + layers * prompt)
    logits = 4.0 * b * VOCAB * (1 if kind == "generate" else passes)
    return {"bytes": passes * weights + kv + logits,
            "flops": 2.0 * layers * per * rows + 4.0 * b * d * pairs + 2.0 * passes * b * VOCAB * d}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 1e-6, "max": 1e-5}        # exact integer sums, then a few float32 products
    if kind in ("likerax", "miborax"):
        return {"rel": 2.5e-2, "max": 0.15}      # bf16 operands through six layers
    if case["terms"] == 3:
        return {"rel": 2e-5, "max": 2e-4}        # float-faithful activations through float32 norms and sums
    if kind == "ffn":
        return {"rel": 4e-3, "max": 0.1}         # a float32 norm in front of an int8 quantiser: ties may fall either way
    return {"rel": 3e-2, "max": 0.3}             # the same through every layer


# ------------------------------------------------------------------ the paths in float64
def linear64(x, w, scale, terms):
    """x W^T scale; with one term the rows are first rounded to 127 steps of their largest magnitude."""
    w = w.double()
    if terms != 1:
        return x @ w.T * scale
    s = x.abs().amax(-1, keepdim=True) / 127
    s = torch.where(s > 0, s, torch.ones_like(s))
    return (x / s).round().clamp(-128, 127) @ w.T * (s * scale)


def rms64(x, weight, eps):
    x = x / (x.square().mean(-1, keepdim=True) + eps).sqrt()
    return x if weight is None else x * weight.to(x.device, torch.float64)


def ffn64(x, mats, norm, terms):
    gate, up = (linear64(x, *m, terms) for m in mats[:2])
    if terms == 1:
        y = gate.clamp(min=0).square() * up
    else:
        y = gate * torch.nn.functional.silu(up.clamp(-20, 20))
    return linear64(rms64(y, norm, EPS[terms]), *mats[2], terms)


def rotary64(x, first, base, half_split):
    n = x.shape[-1]
    f = base ** (-2.0 * torch.arange(n // 2, device="cuda", dtype=torch.float64) / n)
    a = (first + torch.arange(x.shape[-2], device="cuda", dtype=torch.float64))[:, None] * f
    c, s = a.cos(), a.sin()
    if half_split:
        u, v = x[..., :n // 2], x[..., n // 2:]
        return torch.cat([u * c - v * s, v * c + u * s], -1)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def softmax64(q, k, v, scale, see, bias=None, sink=None):
    """q [heads, n, D], k [heads, t, D], v [heads, t, V]; see [n, t] or None."""
    s = q @ k.transpose(-1, -2) * scale
    if bias is not None:
        s = s + bias
    if see is not None:
        s = s.masked_fill(~see, -math.inf)
    if sink is not None:
        s = torch.cat([s, sink.double()[:, None, None].expand(-1, s.shape[1], 1)], -1)
    p = s.softmax(-1)
    return (p if sink is None else p[..., :-1]) @ v


def positions(first, n, total):
    return torch.arange(first, first + n, device="cuda")[:, None], torch.arange(total, device="cuda")[None]


class Ternary64:
    """The ternary model, one call per portion of tokens."""

    def __init__(self, case, seed):
        self.case, self.sem_terms = case, case["terms"]
        self.layers = [ternary_layer(case, seed, i) for i in range(case["layers"])]
        self.embed = ternary_embedding(case, seed)
        self.caches = [None] * case["layers"]
        self.past = 0
        if case["kind"] == "steps":
            self.caches = [[t.double() for t in cached_rows(case, seed, i)] for i in range(case["layers"])]
            self.past = case["context"]

    def __call__(self, ids):
        terms, s = self.sem_terms, SHAPES[self.case["shape"]]
        h, hk, hd = s["n_heads"], s["n_kv_heads"], s["d_model"] // s["n_heads"]
        eps = EPS[terms]
        ids = torch.as_tensor(np.ascontiguousarray(ids), device="cuda")
        b, n = ids.shape
        x = self.embed[ids].double()
        for i, (mats, norms) in enumerate(self.layers):
            norms = {k: torch.from_numpy(v).cuda().double() for k, v in norms.items()}
            u = rms64(x, norms["input"], eps)
            q, k, v = (linear64(u, *mats[m], terms).reshape(b, n, -1, hd).transpose(1, 2) for m in "qkv")
            if terms == 1:
                q, k = (rotary64(t, self.past, THETA, True) for t in (q, k))
            if self.caches[i] is not None:
                k, v = (torch.cat([c, t], 2) for c, t in zip(self.caches[i], (k, v)))
            if self.case["kind"] != "prompt":
                self.caches[i] = [k, v]
            a, t = positions(self.past, n, self.past + n)
            see = a >= t if terms == 1 else None
            out = torch.stack([softmax64(q[j], k[j].repeat_interleave(h // hk, 0), v[j].repeat_interleave(h // hk, 0), hd ** -0.5, see)
                               for j in range(b)])
            o = linear64(out.transpose(1, 2).reshape(b, n, h * hd), *mats["o"], terms)
            x = x + rms64(o, norms["attn"], eps)
            x = x + ffn64(rms64(x, norms["post"], eps), [mats[m] for m in ("gate", "up", "down")], norms["ffn"], terms)
        self.past += n
        return rms64(x[:, -1], None, eps) @ self.embed.double().T


def likerax64(case, seed):
    c = LIKERAX
    g = generator(seed, 6)
    embed, head = dense(g, c["vocab"], c["d"]) * c["d"] ** 0.5, dense(g, c["vocab"], c["d"])
    prompt, steps = tokens(case, seed, c["vocab"])
    ids = torch.as_tensor(np.concatenate([prompt] + list(steps), 1), device="cuda")
    b, n = ids.shape
    x = embed[ids].double()
    streams = [x.clone() for _ in range(c["streams"])]
    a, t = positions(0, n, n)
    see = (t <= a) & (a // c["chunk"] == t // c["chunk"])
    slopes = torch.tensor([2.0 ** (-8.0 * (i + 1) / c["heads"]) for i in range(c["heads"])], device="cuda", dtype=torch.float64)
    bias = -(a - t).double()
    for i in range(case["layers"]):
        w = likerax_layer(seed, i)
        mat = lambda z, name: z @ w[name].double().T
        for part in (1, 2):
            u = sum(float(w[f"in{part}"][s]) * streams[s] for s in range(c["streams"]))
            u = rms64(u, w[f"norm{part}"], 1e-5)
            if part == 1:
                split = lambda z, m: z.reshape(b, n, m, c["dim"]).transpose(1, 2)
                q, k, v = split(mat(u, "q"), c["heads"]), split(mat(u, "k"), c["kv"]), split(mat(u, "v"), c["kv"])
                q, k = rms64(q, None, 1e-5), rms64(k, None, 1e-5)
                r = c["heads"] // c["kv"]
                out = torch.stack([torch.cat([softmax64(q[j, hh:hh + 1], k[j, hh // r:hh // r + 1], v[j, hh // r:hh // r + 1], c["dim"] ** -0.5,
                                                        see, slopes[hh] * bias) for hh in range(c["heads"])]) for j in range(b)])
                y = mat(out.transpose(1, 2).reshape(b, n, -1), "o")
            else:
                y = mat(torch.nn.functional.gelu(mat(u, "gate"), approximate="tanh") * mat(u, "up"), "down")
            mix, give = w[f"mix{part}"], w[f"out{part}"]
            streams = [sum(float(mix[s, k2]) * streams[s] for s in range(c["streams"])) + float(give[k2]) * y for k2 in range(c["streams"])]
    last = sum(streams)[:, case["context"] - 1 + (1 if case["steps"] else 0):]
    return [rms64(last[:, j], None, 1e-5) @ head.double().T for j in range(last.shape[1])]


def miborax64(case, seed):
    c = MIBORAX
    embed = miborax_embedding(seed)
    prompt, steps = tokens(case, seed, c["vocab"])
    ids = torch.as_tensor(np.concatenate([prompt] + list(steps), 1), device="cuda")
    b, n = ids.shape
    x = embed[ids].double() * c["d"] ** 0.5
    a, t = positions(0, n, n)
    rows = None

    def norm(z):
        z = z - z.mean(-1, keepdim=True)
        return z / (z.square().mean(-1, keepdim=True) + 1e-5).sqrt()

    for i in range(case["layers"]):
        w, full, lent = miborax_layer(seed, i)
        mat = lambda z, m: z @ m.double().T
        u = norm(x)
        if not lent:
            z = mat(u, w["dkv"])
            rows = rms64(z[..., :c["rank"]], None, 1e-5), rotary64(z[..., c["rank"]:], 0, 10000.0, False)
        q = mat(rms64(mat(u, w["dq"]), None, 1e-5), w["uq"]) if full else mat(u, w["q"])
        q = q.reshape(b, n, c["heads"], -1).transpose(1, 2)
        q = torch.cat([q[..., :c["dim"]], rotary64(q[..., c["dim"]:], 0, 10000.0, False)], -1)
        k, v = (mat(rows[0], w[m]).reshape(b, n, c["heads"], -1).transpose(1, 2) for m in ("uk", "uv"))
        k = torch.cat([k, rows[1][:, None].expand(-1, c["heads"], -1, -1)], -1)
        see = (t <= a) if full else (t <= a) & (a - t < c["window"])
        out = torch.stack([softmax64(q[j], k[j], v[j], (c["dim"] + c["rot"]) ** -0.5, see, sink=w["sink"]) for j in range(b)])
        if full:
            out = out * mat(u, w["gate"]).sigmoid().transpose(1, 2)[..., None]
        y = mat(out.transpose(1, 2).reshape(b, n, -1), w["o"]).reshape(b * n, -1)
        h = u.reshape(b * n, -1)
        best, chosen = mat(h, w["router"]).topk(c["top"], -1)
        weight = best.softmax(-1)
        for e, (gate, up, down) in enumerate(w["experts"]):
            r, slot = (chosen == e).nonzero(as_tuple=True)
            if len(r):
                z = mat(torch.nn.functional.silu(mat(h[r], gate)) * mat(h[r], up), down)
                y.index_add_(0, r, z * weight[r, slot][:, None])
        x = x + y.reshape(b, n, -1)
    last = x[:, case["context"] - 1 + (1 if case["steps"] else 0):]
    return [norm(last[:, j]) @ embed.double().T for j in range(last.shape[1])]


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        return linear64(rows_of(case, seed).double(), *layer_weights(case, seed)[0], case["terms"])
    if kind == "ffn":
        return ffn64(rows_of(case, seed).double(), layer_weights(case, seed), None, case["terms"])
    if kind == "likerax":
        return likerax64(case, seed)
    if kind == "miborax":
        return miborax64(case, seed)
    model = Ternary64(case, seed)
    prompt, steps = tokens(case, seed, VOCAB)
    if kind == "generate":
        logits, new = model(prompt), []
        for _ in range(case["steps"]):
            new.append(logits.argmax(-1, keepdim=True).cpu().numpy())
            logits = model(new[-1])
        return np.concatenate(new, 1), logits
    out = [] if kind == "steps" else [model(prompt)]
    return out + [model(ids) for ids in steps]
