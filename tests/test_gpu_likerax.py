"""GPU: Likerax through the framework against the plain oracle (oracle/likerax_np.py)."""
import ctypes as C
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import likerax_models as M
from oracle import likerax_np as L

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
F32_TOL, BF16_TOL = 2e-5, 3e-2     # of the RMS; every sublayer's rounding included


def rel(got, want):
    """Largest error of a row, relative to that row's RMS (float64)."""
    got, want = np.asarray(got, dtype=np.float64), np.asarray(want, dtype=np.float64)
    return float(np.max(np.sqrt(np.mean((got - want) ** 2, -1)) / np.sqrt(np.mean(want ** 2, -1) + 1e-30)))


def ld(n):
    return (n + 63) // 64 * 64


def dev(a, dtype=None, cols=None):
    """Host array to the device, columns padded with zeros to `cols`."""
    import torch
    a = np.asarray(a)
    if cols is not None and cols != a.shape[-1]:
        a = np.concatenate([a, np.zeros((*a.shape[:-1], cols - a.shape[-1]), dtype=a.dtype)], -1)
    t = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return t.to(getattr(torch, dtype)) if dtype else t


def tol(dtype):
    return F32_TOL if dtype == "float32" else BF16_TOL


# ------------------------------------------------------------------------------- mechanisms
@pytest.mark.parametrize("streams,n,rows", [(1, 64, 3), (2, 100, 5), (3, 1536, 2), (4, 320, 700), (6, 136, 4)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_stream_stage(streams, n, rows, dtype):
    import torch
    from rotor_b200 import abi
    g = np.random.default_rng(streams * 1000 + n)
    x, y = g.standard_normal((rows, streams, n)).astype(np.float32), g.standard_normal((rows, n)).astype(np.float32)
    mix, out, inn = g.standard_normal((streams, streams)), g.standard_normal(streams), g.standard_normal(streams)
    norm, eps = 1 + 0.3 * g.standard_normal(n), 1e-3
    f = lambda a: dev(np.asarray(a, dtype=np.float32))
    xd, yd, nd = dev(x, cols=ld(n)), dev(y, cols=ld(n)), dev(norm.astype(np.float32), cols=ld(n))
    xo = torch.zeros_like(xd)
    h = torch.full((rows, ld(n)), float("nan"), dtype=getattr(torch, dtype), device="cuda")
    args = [f(mix), f(out), f(inn)]
    abi.check(abi.lib.rotor_b200_stream_stage(None, None, 0, abi.ptr(xd), abi.ptr(xo), abi.ptr(yd), abi.ptr(args[0]), abi.ptr(args[1]),
                                              abi.ptr(args[2]), abi.ptr(nd), eps, rows, streams, n, abi.ptr(h),
                                              int(dtype == "float32"), abi.stream()))
    mix, out, inn = (np.asarray(a, dtype=np.float32).astype(np.float64) for a in (mix, out, inn))
    new = L.hyper_connection([x[:, s].astype(np.float64) for s in range(streams)], np.zeros(streams), mix, out, lambda u: y)
    want = L.rms_norm(sum(inn[s] * new[s] for s in range(streams)), norm.astype(np.float32), eps)
    assert rel(xo.cpu().numpy()[:, :, :n], np.stack(new, 1)) < 1e-6
    hh = h.float().cpu().numpy()
    assert rel(hh[:, :n], want) < (1e-6 if dtype == "float32" else 4e-3)
    assert not hh[:, n:].any()


def test_stream_stage_embedding_fills_every_stream():
    import torch
    from rotor_b200 import abi
    g = np.random.default_rng(7)
    table, ids = M.bf16(g.standard_normal((23, 72))), np.array([5, 22, 0], dtype=np.int64)
    td, idd, one = dev(table, "bfloat16", ld(72)), dev(ids), dev(np.ones(ld(72), dtype=np.float32))
    inn = dev(np.array([0.5, -2.0], dtype=np.float32))
    xo = torch.empty((3, 2, ld(72)), device="cuda")
    h = torch.empty((3, ld(72)), device="cuda")
    abi.check(abi.lib.rotor_b200_stream_stage(abi.ptr(idd), abi.ptr(td), 23, None, abi.ptr(xo), None, None, None, abi.ptr(inn),
                                              abi.ptr(one), 1e-6, 3, 2, 72, abi.ptr(h), 1, abi.stream()))
    assert np.array_equal(xo.cpu().numpy()[:, :, :72], np.repeat(table[ids][:, None], 2, 1))
    assert rel(h.cpu().numpy()[:, :72], L.rms_norm(-1.5 * table[ids], None, 1e-6)) < 1e-6


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 33, 130, 700])
@pytest.mark.parametrize("n,k", [(48, 64), (200, 136), (1000, 776), (7, 2100)])
@pytest.mark.parametrize("gated", [0, 1])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_dense_linear(rows, n, k, gated, dtype):
    _dense(rows, n, k, gated, dtype)


@pytest.mark.parametrize("rows,n,k,gated", [(2600, 2000, 200, 0), (2600, 1100, 136, 1), (5000, 4224, 96, 0)])
def test_dense_linear_more_tiles_than_sms(rows, n, k, gated):
    _dense(rows, n, k, gated, "bfloat16")


@pytest.mark.parametrize("rows", [3, 5, 25, 26, 31, 32, 33])
@pytest.mark.parametrize("n,k,gated", [(200, 136, 1), (10000, 776, 0), (40, 5000, 0), (5000, 200, 1)])
def test_dense_linear_around_the_small_token_box(rows, n, k, gated):
    _dense(rows, n, k, gated, "bfloat16")


def _dense(rows, n, k, gated, dtype):
    import torch
    from rotor_b200 import abi
    g = np.random.default_rng(rows + n + k)
    w, x = M.bf16(g.standard_normal((n * (1 + gated), k)) / np.sqrt(k)), M.bf16(g.standard_normal((rows, k)))
    wd, xd = dev(w, "bfloat16", ld(k)), dev(x, dtype, ld(k))
    if ld(k) > k:   # what lies in the pad columns of activations must not matter
        xd[:, k:] = 3.0
    y = torch.zeros((rows, ld(n)), dtype=getattr(torch, dtype) if gated else torch.float32, device="cuda")
    scratch = torch.empty((rows, 2 * n), dtype=torch.float32, device="cuda")
    abi.check(abi.lib.rotor_b200_dense_linear(abi.ptr(wd), n, k, abi.ptr(xd), rows, int(dtype == "float32"), gated, abi.ptr(y),
                                              abi.ptr(scratch), abi.stream()))
    abi.device_status()
    want = L.linear(w, x.astype(np.float64))
    if gated:
        want = L.gelu_tanh(want[:, :n]) * want[:, n:]
    assert rel(y.float().cpu().numpy()[:, :n], want) < (4e-3 if gated and dtype == "bfloat16" else 1e-5)


class Attn:
    """Attention of a batch of sequences through the C entry point, caches kept between calls."""

    def __init__(self, heads, kv, dim, vdim, chunk, scale, slopes, dtype, batch=1, max_seq=512, unit=True, eps=1e-6):
        import torch
        from rotor_b200 import abi
        self.h, self.g, self.d, self.v, self.chunk, self.scale, self.slopes = heads, kv, dim, vdim, chunk, scale, slopes
        self.dtype, self.batch, self.max_seq, self.unit, self.eps = dtype, batch, max_seq, unit, eps
        up8 = lambda a: (a + 7) // 8 * 8
        t = getattr(torch, dtype)
        self.kc = torch.zeros((batch, kv, max_seq, up8(dim)), dtype=t, device="cuda")
        self.vc = torch.zeros((batch, kv, max_seq, up8(vdim)), dtype=t, device="cuda")
        self.q_scratch = torch.empty(batch * max_seq * heads * up8(dim), dtype=torch.bfloat16, device="cuda")
        self.sl = dev(np.asarray(slopes, dtype=np.float32)) if slopes is not None else None
        self.c = abi.DecoderLayer(heads=heads, kv_heads=kv, dim=dim, vdim=vdim, unit_qk=int(unit), chunk=chunk, scale=scale,
                                  slopes=abi.ptr(self.sl))

    def run(self, q, k, v, past, row_kernel=0):
        """q [batch, seq, heads, dim] etc.; past [batch]."""
        import torch
        from rotor_b200 import abi
        b, t = q.shape[:2]
        raw = np.concatenate([a.reshape(b * t, -1) for a in (q, k, v)], 1).astype(np.float32)
        rd, pd = dev(raw, cols=ld(raw.shape[1])), dev(np.asarray(past, dtype=np.int32))
        out = torch.full((b * t, ld(self.h * self.v)), 0.0, dtype=getattr(torch, self.dtype), device="cuda")
        abi.check(abi.lib.rotor_b200_bias_attention(C.byref(self.c), self.eps, int(self.dtype == "float32"), abi.ptr(rd), b, t,
                                                    abi.ptr(pd), self.max_seq, abi.ptr(self.kc), abi.ptr(self.vc), abi.ptr(out),
                                                    row_kernel, abi.ptr(self.q_scratch), abi.stream()))
        abi.device_status()
        return out.float().cpu().numpy()[:, :self.h * self.v].reshape(b, t, self.h, self.v)

    def want(self, q, k, v):
        """Oracle over one whole sequence [T, heads, dim] ..."""
        if self.unit:
            q, k = L.rms_norm(q, None, self.eps), L.rms_norm(k, None, self.eps)
        out = [L.attention_head(q[:, a].astype(np.float64), k[:, a // (self.h // self.g)].astype(np.float64),
                                v[:, a // (self.h // self.g)].astype(np.float64), self.scale,
                                0.0 if self.slopes is None else self.slopes[a], self.chunk or None) for a in range(self.h)]
        return np.stack(out, 1)


SHAPES = [  # heads, kv, dim, vdim, chunk
    (4, 2, 64, 64, 40), (8, 1, 32, 96, 24), (6, 2, 128, 128, 150), (3, 3, 80, 40, 0), (5, 1, 20, 24, 33), (12, 4, 64, 128, 64),
    (16, 1, 128, 64, 1), (2, 1, 160, 200, 50), (7, 1, 64, 48, 90), (9, 9, 48, 64, 60), (10, 1, 96, 128, 100)]


@pytest.mark.parametrize("heads,kv,dim,vdim,chunk", SHAPES)
@pytest.mark.parametrize("dtype,row_kernel", [("float32", 1), ("bfloat16", 0), ("bfloat16", 1)])
def test_attention_prompt_portions_and_single_tokens(heads, kv, dim, vdim, chunk, dtype, row_kernel):
    g = np.random.default_rng(heads * dim + chunk)
    t = 171
    q, k, v = (M.bf16(g.standard_normal((t, n, d))) for n, d in ((heads, dim), (kv, dim), (kv, vdim)))
    a = Attn(heads, kv, dim, vdim, chunk, 0.3, [2.0 ** (-8 * (h + 1) / heads) for h in range(heads)], dtype, max_seq=192)
    want = a.want(q, k, v)
    got, at = [], 0
    for n in (90, 2, 17, 1, 1, 40, 3, 1, 1, 1, 14):
        got.append(a.run(q[None, at:at + n], k[None, at:at + n], v[None, at:at + n], [at], row_kernel)[0])
        at += n
    assert at == t
    assert rel(np.concatenate(got).reshape(t, -1), want.reshape(t, -1)) < tol(dtype) / 2


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_attention_of_unequal_sequences_in_one_batch(dtype):
    g = np.random.default_rng(11)
    heads, kv, dim, vdim, chunk = 4, 2, 64, 64, 30
    lens, new = [0, 7, 29, 30, 31, 95, 60], 1
    for new in (1, 20):
        a = Attn(heads, kv, dim, vdim, chunk, 0.25, [0.5, 0.1, 0.02, 0.004], dtype, batch=len(lens), max_seq=128)
        data = [[M.bf16(g.standard_normal((n + new, c, d))) for c, d in ((heads, dim), (kv, dim), (kv, vdim))] for n in lens]
        for b, n in enumerate(lens):   # fill each sequence's cache through its own view of the batch
            if n:
                one = Attn(heads, kv, dim, vdim, chunk, 0.25, a.slopes, dtype, max_seq=128)
                one.run(*(x[None, :n] for x in data[b]), [0])
                a.kc[b], a.vc[b] = one.kc[0], one.vc[0]
        got = a.run(*(np.stack([d[i][-new:] for d in data]) for i in range(3)), lens)
        for b in range(len(lens)):
            want = a.want(*data[b])[-new:]
            assert rel(got[b].reshape(new, -1), want.reshape(new, -1)) < tol(dtype) / 2, (new, b)


@pytest.mark.parametrize("dtype,row_kernel", [("float32", 1), ("bfloat16", 0), ("bfloat16", 1)])
@pytest.mark.parametrize("key,query", [(0, 63), (64, 127), (63, 64), (1, 64), (127, 128), (128, 169), (40, 41), (64, 64), (100, 169)])
def test_one_key_stands_out_inside_and_outside_the_chunk(key, query, dtype, row_kernel):
    """Key `key` points along query `query` alone: visible, it takes the whole weight; in another chunk, none."""
    heads, kv, dim, vdim, chunk, t = 4, 2, 64, 64, 64, 170
    g = np.random.default_rng(key * 200 + query)
    q, k, v = (g.standard_normal((t, n, d)) for n, d in ((heads, dim), (kv, dim), (kv, vdim)))
    k[key, :] = 0
    for a in range(heads):
        k[key, a // 2] += q[query, a] / 2
    q, k, v = M.bf16(q), M.bf16(k), M.bf16(v)
    a = Attn(heads, kv, dim, vdim, chunk, 0.5, [0.02, 0.01, 0.005, 0.001], dtype, max_seq=192)
    want = a.want(q, k, v)
    seen = key // chunk == query // chunk
    near = np.abs(want[query] - np.repeat(v[key], 2, 0)).max()
    assert (near < 0.2) == seen                       # the input shows what it is meant to show
    # as one prompt, and as a decoded token
    got = a.run(q[None], k[None], v[None], [0], row_kernel)[0]
    assert rel(got.reshape(t, -1), want.reshape(t, -1)) < tol(dtype) / 2
    b = Attn(heads, kv, dim, vdim, chunk, 0.5, a.slopes, dtype, max_seq=192)
    if query:
        b.run(q[None, :query], k[None, :query], v[None, :query], [0], row_kernel)
    one = b.run(q[None, query:query + 1], k[None, query:query + 1], v[None, query:query + 1], [query])[0]
    assert rel(one.reshape(1, -1), want[query:query + 1].reshape(1, -1)) < tol(dtype) / 2


@pytest.mark.parametrize("dim,vdim", [(64, 32), (128, 72), (136, 160)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_chunk_decoding_walks_many_tiles(dim, vdim, dtype):
    """A run of keys longer than eight splits of one tile, no unit norm, no bias."""
    heads, kv, t = 4, 1, 2100
    g = np.random.default_rng(5)
    q, k, v = (M.bf16(g.standard_normal((t, n, d))) for n, d in ((heads, dim), (kv, dim), (kv, vdim)))
    k[3] = q[t - 1, 0]      # a key far back that only the last query asks for
    a = Attn(heads, kv, dim, vdim, 0, 0.2, None, dtype, max_seq=2112, unit=False)
    a.run(q[None, :t - 1], k[None, :t - 1], v[None, :t - 1], [0])
    got = a.run(q[None, -1:], k[None, -1:], v[None, -1:], [t - 1])[0, 0]
    for h in range(heads):
        s = (k[:, 0].astype(np.float64) @ q[-1, h].astype(np.float64)) * 0.2
        p = np.exp(s - s.max())
        assert rel(got[h][None], (p @ v[:, 0].astype(np.float64) / p.sum())[None]) < tol(dtype) / 2
    assert np.abs(got[0] - v[3, 0]).max() < 0.5


# ------------------------------------------------------------------------------- whole models
CONFIGS = {
    "mixed": lambda: M.config([M.layer(chunk=24), M.layer(heads=6, kv_heads=2, dim=40, vdim=24, chunk=17, ff=None, scale=0.5),
                               M.layer(heads=2, kv_heads=1, dim=64, vdim=32, chunk=50, ff=200)], loop=(1, 3, 2)),
    "one stream": lambda: M.config([M.layer(heads=4, kv_heads=4, dim=128, vdim=128, chunk=16, ff=128)], streams=1, width=320, vocab=64),
    "four streams": lambda: M.config([M.layer(heads=8, kv_heads=1, dim=64, vdim=64, chunk=37, ff=72, scale=0.2),
                                      M.layer(heads=4, kv_heads=1, dim=64, vdim=64, chunk=37, ff=64)], streams=4, width=256, vocab=300,
                                     loop=(0, 1, 3)),
    "five streams": lambda: M.config([M.layer(chunk=1000), M.layer(chunk=9, ff=None)], streams=5, width=72, vocab=31, eps=1e-3),
}


@pytest.fixture(scope="module")
def case():
    cache = {}

    def get(name, dtype):
        if name not in cache:
            m = M.make(CONFIGS[name](), seed=len(name))
            toks = np.random.default_rng(1).integers(0, m["cfg"]["vocab"], 123)
            cache[name] = (m, toks, L.forward(m, toks))
        m, toks, want = cache[name]
        if (name, dtype) not in cache:
            cache[name, dtype] = M.load(m, dtype=dtype, max_seq=160)
        return cache[name, dtype], m, toks, want
    return get


def feed(model, toks, sizes, start=0):
    """Logits of every position, the tokens cut into portions of the given sizes (repeated)."""
    out, at, i = [], start, 0
    while at < len(toks):
        n = min(sizes[i % len(sizes)], len(toks) - at)
        out.append(model.forward_rows_device(toks[at:at + n], at, list(range(n))).cpu().numpy())
        at, i = at + n, i + 1
    from rotor_b200 import abi
    abi.device_status()
    return np.concatenate(out)


@pytest.mark.parametrize("name", list(CONFIGS))
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("sizes", [[123], [1], [2], [3], [60, 2, 16, 1, 5], [33, 17]], ids=str)
def test_portions_match_the_oracle(case, name, dtype, sizes):
    model, m, toks, want = case(name, dtype)
    assert rel(feed(model, toks, sizes), want) < tol(dtype)


def test_planted_mistakes_would_show(case):
    """The oracle with one mistake each is far outside the tolerance that the product meets."""
    model, m, toks, want = case("mixed", "bfloat16")
    got = feed(model, toks, [123])

    def other(change):
        c = json.loads(json.dumps(m["cfg"]))
        w = dict(m["w"])
        change(c, w)
        return rel(got, L.forward({"cfg": c, "w": w}, toks))

    def chunk(c, w):
        c["layers"][0]["mixer"]["mask"]["size"] += 1

    def transposed(c, w):
        w["l0.hc2.mix"] = w["l0.hc2.mix"].T

    def one_pass(c, w):
        c["loop"]["times"] = 1

    def scale(c, w):
        c["layers"][2]["mixer"]["scale"] *= 1.3

    assert rel(got, want) < BF16_TOL
    for change in (chunk, transposed, one_pass, scale):
        assert other(change) > 3 * BF16_TOL, change.__name__


def test_a_loop_keeps_a_cache_per_pass(case):
    model, m, toks, want = case("four streams", "float32")
    assert len(model.runs) == 4
    feed(model, toks, [50, 1])
    keys = [r.k_cache[0, 0, :len(toks)].cpu().numpy() for r in model.runs]
    assert all(np.abs(keys[0] - keys[i]).max() > 0.1 for i in (1, 2))


def test_positions_that_are_given_back_are_used_again(case):
    model, m, toks, want = case("mixed", "float32")
    other = np.random.default_rng(9).integers(0, m["cfg"]["vocab"], 140)
    feed(model, other, [140])
    assert rel(feed(model, toks[:40], [11, 1, 2]), want[:40]) < F32_TOL
    feed(model, other, [7])
    assert rel(feed(model, toks, [123]), want) < F32_TOL


def test_the_cache_grows_and_keeps_its_contents(case):
    _, m, toks, want = case("mixed", "float32")
    model = M.load(m, dtype="float32", max_seq=16, max_rows=8)
    assert rel(feed(model, toks, [8, 1, 30]), want) < F32_TOL


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_long_decoding_crosses_many_chunks(case, dtype):
    model, m, toks, want = case("four streams", dtype)
    assert rel(feed(model, toks, [5] + [1] * 118), want) < tol(dtype)


def test_api_forward_shapes_and_caches(case):
    model, m, toks, want = case("one stream", "float32")
    both, caches = model.forward(np.stack([toks[:20], toks[20:40]]), use_cache=True)
    assert both.shape == (2, 20, m["cfg"]["vocab"]) and rel(both[0], want[:20]) < F32_TOL
    assert caches[0]["k"].shape == (2, 4, 20, 128)
    step, caches = model.forward(np.array([[toks[20]], [toks[40]]]), past_kv_cache=caches, use_cache=True)
    assert rel(step[0], want[20:21]) < F32_TOL and caches[0].length == 21
    assert rel(step[1], L.forward(m, toks[20:41])[-1:]) < F32_TOL


# ------------------------------------------------------------------------------- generation
def greedy_want(m, prompt, n):
    """Oracle generation and the smallest margin between the two best logits on the way."""
    seq, margin = [int(t) for t in prompt], np.inf
    for _ in range(n):
        lg = L.forward(m, seq)[-1]
        top = np.sort(lg)
        margin = min(margin, (top[-1] - top[-2]) / np.sqrt(np.mean(lg ** 2)))
        seq.append(int(np.argmax(lg)))
    return seq[len(prompt):], margin


def test_greedy_generation_through_the_text_generator(case):
    from rotor_b200.generation import TextGenerator, TopKSampling
    from rotor_b200.synth import PassThroughTokenizer
    model, m, toks, _ = case("mixed", "float32")
    prompt, n = toks[:21], 30
    want, margin = greedy_want(m, prompt, n)
    assert margin > 10 * F32_TOL
    for use_cache in (True, False):
        gen = TextGenerator(model, PassThroughTokenizer(), max_length=len(prompt) + n, use_cache=use_cache)
        out = [int(t) for t in gen.generate(" ".join(map(str, prompt)), max_new_tokens=n, stop_on_eos=False).split()]
        assert out[len(prompt):] == want
    assert model.generate_greedy(prompt, n, use_graph=False) == want
    # a draw among one candidate is the greedy pick, through the device sampler
    gen = TextGenerator(model, PassThroughTokenizer(), TopKSampling(1, seed=3), max_length=len(prompt) + n)
    out = [int(t) for t in gen.generate(" ".join(map(str, prompt)), max_new_tokens=n, stop_on_eos=False).split()]
    assert out[len(prompt):] == want


@pytest.mark.parametrize("lens", [[3, 21, 24, 48], [1, 30, 17, 2, 64, 25, 23]], ids=["fused step", "seven prompts"])
def test_batch_of_unequal_prompts_generates_what_each_does_alone(case, lens):
    model, m, toks, _ = case("mixed", "float32")
    prompts = [toks[i:i + n] for i, n in enumerate(lens)]
    got = model.generate_greedy_batch(prompts, 12)
    for b, p in enumerate(prompts):
        want, margin = greedy_want(m, p, 12)
        assert margin > 10 * F32_TOL
        assert got[b].tolist() == want, b
    same = model.generate_greedy_batch([prompts[1]] * 3, 12)
    assert all(r.tolist() == got[1].tolist() for r in same)


def test_unfused_steps_give_the_same_tokens(case):
    """ROTOR_B200_NO_FUSED_STEP: stages and products as kernels of their own."""
    model, m, toks, want = case("four streams", "bfloat16")
    code = ("import sys, numpy as np, likerax_models as M, test_gpu_likerax as T\n"
            "m = M.make(T.CONFIGS['four streams'](), seed=len('four streams'))\n"
            "toks = np.random.default_rng(1).integers(0, m['cfg']['vocab'], 123)\n"
            "np.save(sys.argv[1], T.feed(M.load(m, max_seq=160), toks, [60, 1, 3]))\n")
    out = os.path.join(os.environ.get("TMPDIR", "/tmp"), f"likerax_unfused_{os.getpid()}.npy")
    env = dict(os.environ, ROTOR_B200_NO_FUSED_STEP="1",
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "rotor-rag_b200"), os.path.join(ROOT, "tests")]))
    try:
        subprocess.check_call([sys.executable, "-c", code, out], env=env, cwd=ROOT)
        got = np.load(out)
    finally:
        if os.path.exists(out):
            os.remove(out)
    assert rel(got, want) < BF16_TOL


# ------------------------------------------------------------------------------- files and programs
def test_checkpoint_command_line_and_trace_replay(tmp_path, case, capsys):
    from rotor_b200.__main__ import main
    _, m, toks, want = case("mixed", "float32")
    folder = M.write(m, tmp_path / "model")
    prompt = " ".join(str(int(t)) for t in toks[:21])
    assert main(["generate", "--model", folder, "--dtype", "float32", "--prompt", prompt, "--max-new-tokens", "10"]) == 0
    assert [int(t) for t in capsys.readouterr().out.split()] == greedy_want(m, toks[:21], 10)[0]

    steps = [{"step": 0, "entries": [{"id": "a", "tokens": toks[:70].tolist(), "want": [0, 23, 24, 69]}], "end": []},
             {"step": 1, "entries": [{"id": "a", "tokens": toks[70:73].tolist(), "want": []}], "end": []},
             {"step": 2, "entries": [{"id": "a", "tokens": toks[73:74].tolist(), "want": [0]}], "end": ["a"]},
             {"step": 3, "entries": [{"id": "b", "tokens": toks[:30].tolist(), "want": [29, 1]}], "end": ["b"]}]
    rows = {0: [0, 23, 24, 69], 2: [73], 3: [29, 1]}
    for dtype in ("bfloat16", "float32"):
        out = tmp_path / dtype
        out.mkdir()
        r = subprocess.run([os.path.join(ROOT, "bin", "trace_run"), "--model", folder, "--dtype", dtype, "--out", str(out),
                            "--max-tokens", "80"], input="\n".join(json.dumps(s) for s in steps), capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
        assert r.stdout.split("\n")[:4] == [f"done {i}" for i in range(4)]
        assert not (out / "1.f32").exists()
        for i, at in rows.items():
            got = np.fromfile(out / f"{i}.f32", dtype="<f4").reshape(len(at), -1)
            assert rel(got, want[at]) < tol(dtype)
