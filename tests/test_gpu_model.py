"""GPU: the decode path above BitLinear (a6-a12) through the reference-shaped Python API,
against the fixtures produced by the unmodified reference and against the oracle.
Tolerance for floating outputs: max-abs error below 1e-3 of the output RMS."""
import os

import numpy as np
import pytest

import golden_inputs as G
from oracle import bitlinear_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-3


def rel_err(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.max(np.abs(a - b)) / np.sqrt(np.mean(b ** 2)))


@pytest.fixture(scope="module")
def rb():
    import rotor_b200.transformer as tr
    import rotor_b200.bitnet_model as bm
    import rotor_b200.generation as gen
    import rotor_b200.synth as synth
    from rotor_b200 import semantics
    class NS: pass
    ns = NS()
    ns.tr, ns.bm, ns.gen, ns.synth, ns.sem = tr, bm, gen, synth, semantics
    return ns


def o_sem(s):
    """rotor_b200 semantics -> oracle semantics (three-term int8 stands for the float path)."""
    return O.Semantics(act_terms=0 if s.act_terms == 3 else s.act_terms, ffn_act=s.ffn_act,
                       rope_theta=s.rope_theta, causal=s.causal, eps=s.eps)


def test_rmsnorm(rb):
    rng = np.random.default_rng(0)
    x = rng.standard_normal((3, 5, 2560)).astype(np.float32)
    n = rb.tr.RMSNorm(2560)
    n.weight = 1.0 + 0.1 * rng.standard_normal(2560).astype(np.float32)
    assert rel_err(n.forward(x), O.rmsnorm(x, n.weight, 1e-6)) < 1e-5


def test_ternary_linear_api(rb, golden_dir):
    """TernaryLinear with the reference's call pattern (examples/test_gpu_layer.py:34-46)."""
    z = np.load(os.path.join(golden_dir, "bitlinear_2560x6912.npz"))
    w, scale, x1, x16 = G.bitlinear_case()
    lin = rb.tr.TernaryLinear(2560, 6912, use_gpu=True)
    assert lin.weights_cache is None
    lin.load_from_bitnet(O.pack_ternary_matrix(w), scale)
    assert lin.in_features == 2560 and lin.out_features == 6912 and lin.scale == scale
    assert np.array_equal(lin.weights_cache, w)
    assert rel_err(lin.forward(x1), z["y1"]) < TOL
    y = lin.forward(x16.reshape(2, 8, 2560))          # 3-D input keeps its leading dims
    assert y.shape == (2, 8, 6912) and rel_err(y.reshape(16, -1), z["y16"]) < TOL
    with pytest.raises(Exception):
        rb.tr.TernaryLinear(8, 8, use_gpu=False)       # no CPU path
    with pytest.raises(Exception):
        rb.tr.TernaryLinear(128, 16).forward(np.zeros((1, 128), np.float32))   # never loaded
    with pytest.raises(ValueError):
        lin.load_from_bitnet(np.zeros((4, 4), np.uint8), 1.0)


@pytest.mark.parametrize("mode", ["reference", "baseline"])
def test_ffn_block_config2(rb, golden_dir, mode):
    """Config 2: RMSNorm(2560) -> gate/up -> gating -> sub-norm(6912) -> down, batch 1 and 16."""
    z = np.load(os.path.join(golden_dir, "ffn_block.npz"))
    lw, x1, x16 = G.ffn_case()
    sem = rb.sem.REFERENCE if mode == "reference" else rb.sem.BASELINE
    ffn = rb.tr.GatedFFN(2560, 6912, semantics=sem)
    pre = rb.tr.RMSNorm(2560, eps=sem.eps)
    pre.weight = lw["post_attn_norm"]
    ffn.ffn_norm.weight = lw["ffn_sub_norm"]
    for nm, proj in (("gate", ffn.gate_proj), ("up", ffn.up_proj), ("down", ffn.down_proj)):
        proj.load_from_bitnet(O.pack_ternary_matrix(lw[nm][0]), lw[nm][1])
    from rotor_b200 import ops
    import torch
    for tag, x in (("m1", x1), ("m16", x16)):
        y_fused = ffn.forward_device(ops.to_device(x, torch.float32), pre_norm=pre).cpu().numpy()
        y_api = ffn.forward(pre.forward(x))
        want = O.ffn(O.rmsnorm(x, lw["post_attn_norm"], sem.eps), lw, o_sem(sem))
        if mode == "reference":
            assert rel_err(y_fused, z[tag]) < TOL and rel_err(y_api, z[tag]) < TOL
        assert rel_err(y_fused, want) < TOL, (mode, tag, rel_err(y_fused, want))
        assert rel_err(y_api, want) < TOL


@pytest.mark.parametrize("rows", [1, 2, 3])
def test_ffn_large_matrix_variants(rb, rows):
    """An FFN big enough (2048 -> 2 x 20480 -> 2048) that the generation-step products take their
    large-matrix variants: the pipelined tile loop (eight or more weight tiles per warp) and, for the
    20480-wide input of the down projection, the shared-memory prologue.  One, two and three rows
    select the one-column DP4A, two-column DP4A and tensor-core tile products."""
    import torch
    from rotor_b200 import ops
    d, ff = 2048, 20480
    rng = np.random.default_rng(1000 + rows)
    lw = {"gate": (O.synth_ternary(rng, ff, d), 0.017), "up": (O.synth_ternary(rng, ff, d), 0.015),
          "down": (O.synth_ternary(rng, d, ff), 0.016),
          "ffn_sub_norm": (1.0 + 0.1 * rng.standard_normal(ff)).astype(np.float32)}
    pre_w = (1.0 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    sem = rb.sem.BASELINE
    ffn = rb.tr.GatedFFN(d, ff, semantics=sem)
    pre = rb.tr.RMSNorm(d, eps=sem.eps)
    pre.weight = pre_w
    ffn.ffn_norm.weight = lw["ffn_sub_norm"]
    for nm, proj in (("gate", ffn.gate_proj), ("up", ffn.up_proj), ("down", ffn.down_proj)):
        proj.load_from_int8(lw[nm][0], lw[nm][1])
    before = rb.tr.abi.lib.rotor_b200_launch_count()
    got = ffn.forward_device(ops.to_device(x, torch.float32), pre_norm=pre).cpu().numpy()
    assert rb.tr.abi.lib.rotor_b200_launch_count() - before == 2     # the fused two-launch route
    want = O.ffn(O.rmsnorm(x, pre_w, sem.eps), lw, o_sem(sem))
    assert rel_err(got, want) < TOL, rel_err(got, want)
    rb.tr.abi.device_status()


def _tiny(rb, name, sem, **kw):
    om, prompt = G.tiny_model(name)
    kw.setdefault("max_seq", 64)
    return om, prompt, rb.synth.model_from_oracle_params(om, semantics=sem, **kw)


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
def test_attention_and_block_standalone(rb, name):
    om, prompt, model = _tiny(rb, name, rb.sem.REFERENCE)
    cfg, lw = om["cfg"], om["layers"][0]
    rng = np.random.default_rng(5)
    x = rng.standard_normal((1, 6, cfg["d_model"])).astype(np.float32)
    blk = model.layers[0]
    want, wc = O.attention(x, lw, cfg, O.REFERENCE, None, True)
    got, cache = blk.attention.forward(x, use_cache=True)
    assert rel_err(got, want) < TOL
    assert rel_err(cache["k"], wc["k"]) < TOL and rel_err(cache["v"], wc["v"]) < TOL
    # one more token against the cache
    x2 = rng.standard_normal((1, 1, cfg["d_model"])).astype(np.float32)
    want2, _ = O.attention(x2, lw, cfg, O.REFERENCE, wc, True)
    got2, cache2 = blk.attention.forward(x2, kv_cache=cache, use_cache=True)
    assert rel_err(got2, want2) < TOL and cache2.length == 7
    # whole block, 2-D input like the reference accepts
    wantb, _ = O.block(x, lw, cfg, O.REFERENCE)
    gotb, none = blk.forward(x[0])
    assert none is None and gotb.shape == x[0].shape and rel_err(gotb, wantb[0]) < TOL
    # causal mask through the mask argument
    mask = O.causal_mask(6, 6)
    wantc, _ = O.block(x, lw, cfg, O.with_semantics(O.REFERENCE, causal=True))
    gotc, _ = blk.forward(x, mask=mask)
    assert rel_err(gotc, wantc) < TOL
    with pytest.raises(NotImplementedError):
        blk.forward(x, mask=np.zeros((6, 6)) + 1.0)


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
def test_model_forward_matches_reference_fixture(rb, golden_dir, name):
    z = np.load(os.path.join(golden_dir, f"model_{name}.npz"))
    om, prompt, model = _tiny(rb, name, rb.sem.REFERENCE)
    logits, caches = model.forward(prompt[None, :], use_cache=True)
    assert logits.shape == z["prompt_logits"][None].shape
    assert rel_err(logits[0], z["prompt_logits"]) < TOL
    assert len(caches) == om["cfg"]["n_layers"]
    assert rel_err(caches[-1]["k"], z["last_k"]) < TOL
    l1, _ = model.forward(prompt)                      # 1-D ids -> [S, V]
    assert l1.shape == z["prompt_logits"].shape and rel_err(l1, z["prompt_logits"]) < TOL
    last, _ = model.forward(prompt[None, :], logits_positions="last")
    assert rel_err(last[0, -1], z["prompt_logits"][-1]) < TOL
    hid, _ = model.forward(prompt[None, :], return_logits=False)
    want_h, _ = O.model_forward(om, prompt[None, :], O.REFERENCE, return_logits=False)
    assert rel_err(hid, want_h) < TOL
    mc = rb.synth.model_from_oracle_params(om, semantics=rb.sem.REFERENCE.with_(causal=True), max_seq=64)
    lc, _ = mc.forward(prompt[None, :])
    assert rel_err(lc[0], z["prompt_logits_causal"]) < TOL


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
def test_greedy_generation_identical_to_reference(rb, golden_dir, name):
    """First 32 greedy tokens equal the reference's (TextGenerator, use_cache=True), through the
    device-resident graph path, the eager step path, and the host-sampling path."""
    z = np.load(os.path.join(golden_dir, f"model_{name}.npz"))
    om, prompt, model = _tiny(rb, name, rb.sem.REFERENCE)
    want = z["greedy_ids"].tolist()
    n_new = len(want) - len(prompt)
    assert n_new == G.N_NEW
    tok = rb.synth.PassThroughTokenizer()
    text = " ".join(map(str, prompt))
    tg = rb.gen.TextGenerator(model, tok, max_length=len(want), use_cache=True)
    seen = []
    out = tg.generate(text, max_new_tokens=n_new, stop_on_eos=False, callback=seen.append)
    assert [int(t) for t in out.split()] == want
    assert [int(t) for t in seen] == want[len(prompt):]
    assert model.generate_greedy(prompt, n_new, use_graph=False) == want[len(prompt):]
    assert model.generate_greedy(prompt, n_new, use_graph=True, chunk=0) == want[len(prompt):]
    # host-side sampling strategy object -> logits come back each step
    class Argmax(rb.gen.SamplingStrategy):
        def sample(self, logits, temperature=1.0):
            return int(np.argmax(logits))
    tg2 = rb.gen.TextGenerator(model, tok, sampling_strategy=Argmax(), max_length=len(want), use_cache=True)
    out2 = tg2.generate(text, max_new_tokens=n_new, stop_on_eos=False)
    assert [int(t) for t in out2.split()] == want
    # per-step logits stay within tolerance of the reference's
    logits, cache = model.forward(prompt[None, :], use_cache=True, logits_positions="last")
    assert rel_err(logits[0, -1], z["step_logits"][0]) < TOL
    l2, cache = model.forward(np.array([[want[len(prompt)]]]), past_kv_cache=cache, use_cache=True)
    assert rel_err(l2[0, -1], z["step_logits"][1]) < TOL


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
def test_per_step_logits_against_fixture_margins(rb, golden_dir, name):
    """Every one of the 32 teacher-forced generation steps against the reference fixture: the logit error
    (max-abs over the vocabulary, in units of the step's logit RMS) stays below the tolerance AND below half
    the reference's own top-1 / top-2 margin at that step (stored with the fixture), which is what makes the
    greedy tokens identical rather than merely likely to be."""
    z = np.load(os.path.join(golden_dir, f"model_{name}.npz"))
    om, prompt, model = _tiny(rb, name, rb.sem.REFERENCE)
    want = z["greedy_ids"].tolist()
    logits, cache = model.forward(prompt[None, :], use_cache=True)
    cur = logits[0, -1]
    worst = 0.0
    for i in range(G.N_NEW):
        e = rel_err(cur, z["step_logits"][i])
        worst = max(worst, e)
        assert e < TOL, (i, e)
        assert 2 * e < z["top2_margin"][i], (i, e, float(z["top2_margin"][i]))
        assert int(np.argmax(cur)) == want[len(prompt) + i]
        if i + 1 < G.N_NEW:
            nxt, cache = model.forward(np.array([[want[len(prompt) + i]]]), past_kv_cache=cache, use_cache=True)
            cur = nxt[0, -1]
    print(f"{name}: worst per-step logit error {worst:.2e} of RMS, smallest margin {float(z['top2_margin'].min()):.2e}")


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
def test_baseline_semantics_against_oracle(rb, name):
    """Published semantics (int8 activations, relu^2, rotary, causal, eps 1e-5) against the oracle that
    quantises identically.  A value on a rounding tie of the quantiser is decided by float summation
    order, so the check is tie-aware: the first position (one key, no order-dependent sum before a
    quantiser) within tolerance; every teacher-forced step picks the oracle's token unless the
    oracle's top-2 margin there is below twice the logit error measured at that step; no step
    drifts beyond what flipped ties explain."""
    om, prompt, model = _tiny(rb, name, rb.sem.BASELINE)
    want_logits, _ = O.model_forward(om, prompt[None, :], O.BASELINE)
    logits, cache = model.forward(prompt[None, :], use_cache=True)
    assert rel_err(logits[0, 0], want_logits[0, 0]) < TOL
    assert rel_err(logits, want_logits) < 0.3
    ids, steps = O.generate_greedy(om, prompt, 32, O.BASELINE, return_logits=True)
    want = ids[len(prompt):]
    cur = logits[0, -1]
    equal = 0
    for i in range(32):
        ref = np.asarray(steps[i], np.float64)
        e = rel_err(cur, ref)
        top2 = np.partition(ref, -2)[-2:]
        margin = float((top2[1] - top2[0]) / np.sqrt(np.mean(ref ** 2)))
        assert e < 0.3, (i, e)
        assert int(np.argmax(cur)) == want[i] or margin < 2 * max(e, TOL), (i, int(np.argmax(cur)), want[i], margin, e)
        equal += int(np.argmax(cur)) == want[i]
        if i < 31:
            nxt, cache = model.forward(np.array([[want[i]]]), past_kv_cache=cache, use_cache=True)
            cur = nxt[0, -1]
    assert equal >= 24, equal


def test_generation_loop_rules(rb):
    """max_length caps prompt + new tokens, EOS stops without being appended, streaming yields
    the prompt first (reference src/rotor/generation.py:210, 228-229, 315)."""
    om, prompt, model = _tiny(rb, "hd64", rb.sem.REFERENCE)
    tok = rb.synth.PassThroughTokenizer()
    text = " ".join(map(str, prompt))
    full = model.generate_greedy(prompt, 12)
    tg = rb.gen.TextGenerator(model, tok, max_length=len(prompt) + 4)
    assert len(tg.generate(text, max_new_tokens=50, stop_on_eos=False).split()) == len(prompt) + 4
    tg0 = rb.gen.TextGenerator(model, tok, max_length=len(prompt))
    assert tg0.generate(text) == text                      # nothing to generate
    tok_eos = rb.synth.PassThroughTokenizer(eos_token_id=full[3])
    tg_eos = rb.gen.TextGenerator(model, tok_eos, max_length=64)
    out = [int(t) for t in tg_eos.generate(text, max_new_tokens=12).split()]
    assert out == list(prompt) + full[:full.index(full[3])]
    pieces = list(rb.gen.TextGenerator(model, tok, max_length=64).generate_streaming(text, max_new_tokens=5,
                                                                                   stop_on_eos=False))
    assert pieces[0] == text and [int(p) for p in pieces[1:]] == full[:5]
    # top-k / top-p return valid ids on both routes: drawn on the device (the default with this model) and,
    # with device=False, from host logits with NumPy's global stream as in the reference
    np.random.seed(0)
    assert rb.gen.TopKSampling(k=5).device is None and rb.gen.TopPSampling(p=0.8, device=False).device is False
    for strat in (rb.gen.TopKSampling(k=5), rb.gen.TopPSampling(p=0.8), rb.gen.TopKSampling(k=5, device=False),
                  rb.gen.TopPSampling(p=0.8, device=False)):
        tgs = rb.gen.TextGenerator(model, tok, sampling_strategy=strat, temperature=0.7, max_length=64)
        ids = [int(t) for t in tgs.generate(text, max_new_tokens=4, stop_on_eos=False).split()]
        assert len(ids) == len(prompt) + 4 and all(0 <= t < om["cfg"]["vocab_size"] for t in ids)


def test_load_bitnet_model_from_checkpoint(rb, tmp_path, golden_dir):
    """load_bitnet_model(dir, use_gpu=True) on a synthetic config.json + model.safetensors."""
    z = np.load(os.path.join(golden_dir, "model_hd64.npz"))
    om, prompt = G.tiny_model("hd64")
    rb.synth.write_checkpoint(om, str(tmp_path))
    model = rb.bm.load_bitnet_model(str(tmp_path), use_gpu=True, max_seq=64)
    logits, _ = model.forward(prompt[None, :])
    assert rel_err(logits[0], z["prompt_logits"]) < TOL
    with pytest.raises(Exception):
        rb.bm.load_bitnet_model(str(tmp_path), use_gpu=False)


def test_plugin_backend_object(rb):
    """get_gpu() -> pack_ternary_weights / ternary_matmul with the reference's argument shapes
    (src/rotor/transformer.py:107-109, 136-142)."""
    from rotor_b200.gpu_layers import get_gpu
    gpu = get_gpu()
    assert gpu is get_gpu()
    rng = np.random.default_rng(12)
    w = O.synth_ternary(rng, 2560, 2560)
    packed = gpu.pack_ternary_weights(w)
    scales = np.full(2560, 1.2, dtype=np.float32)
    x = rng.standard_normal(2560).astype(np.float32)
    y = gpu.ternary_matmul(packed, scales, x, 2560, 2560)
    want = (w.astype(np.float32) @ x) * scales
    assert y.dtype == np.float32 and y.shape == (2560,)
    assert np.abs(y - want).max() < 1e-2          # the authors' own GPU-vs-CPU gate (gpu_layers.py:181)
    assert rel_err(y, want) < TOL
    with pytest.raises(ValueError):
        gpu.ternary_matmul(packed, scales, x, 2560, 100)


def test_batched_forward_and_cache_growth(rb):
    om, prompt, model = _tiny(rb, "hd64", rb.sem.REFERENCE, max_batch=1)
    rng = np.random.default_rng(3)
    ids = rng.integers(0, om["cfg"]["vocab_size"], size=(3, 7))
    want, _ = O.model_forward(om, ids, O.REFERENCE)
    got, caches = model.forward(ids, use_cache=True)        # batch 3 > max_batch 1: handle regrows
    assert rel_err(got, want) < TOL and caches[0]["k"].shape[0] == 3
    long_ids = rng.integers(0, om["cfg"]["vocab_size"], size=(1, 90))   # > max_seq 64
    want2, _ = O.model_forward(om, long_ids, O.REFERENCE)
    got2, _ = model.forward(long_ids)
    assert rel_err(got2, want2) < TOL


def test_prefill_and_stepwise_decode_agree(rb):
    """Size-independent property of the cached path (causal semantics): the last-position logits
    of one forward over n+1 tokens equal those of a forward over n tokens followed by a one-token
    step.  The prefill side runs the tiled tensor-core GEMM (>= 32 columns), the step the fused
    generation kernels."""
    om, prompt, model = _tiny(rb, "hd128", rb.sem.BASELINE, max_rows=64)
    rng = np.random.default_rng(17)
    ids = rng.integers(0, om["cfg"]["vocab_size"], size=(1, 41))
    full, _ = model.forward(ids, logits_positions="last")
    _, cache = model.forward(ids[:, :40], use_cache=True, logits_positions="last")
    step, _ = model.forward(ids[:, 40:], past_kv_cache=cache, use_cache=True, logits_positions="last")
    # int8 rounding decisions can differ between the two routes only through float32 summation order
    assert rel_err(step[0, -1], full[0, -1]) < 2e-2
    ref = rb.synth.model_from_oracle_params(om, semantics=rb.sem.REFERENCE.with_(causal=True), max_seq=64)
    full_r, _ = ref.forward(ids, logits_positions="last")
    _, cache_r = ref.forward(ids[:, :40], use_cache=True, logits_positions="last")
    step_r, _ = ref.forward(ids[:, 40:], past_kv_cache=cache_r, use_cache=True, logits_positions="last")
    assert rel_err(step_r[0, -1], full_r[0, -1]) < TOL


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
@pytest.mark.parametrize("causal", [False, True])
def test_tiled_prefill_attention(rb, name, causal):
    """Prompts of 16 positions and more take the tiled attention kernel: ragged lengths (not a
    multiple of the 64-key tile or of the query tile), batch 2, then a second chunk attending
    over the cached keys of the first."""
    sem = rb.sem.REFERENCE.with_(causal=causal)
    osem = O.with_semantics(O.REFERENCE, causal=causal)
    om, prompt, model = _tiny(rb, name, sem, max_seq=256, max_batch=2)
    cfg, lw = om["cfg"], om["layers"][0]
    rng = np.random.default_rng(23)
    att = model.layers[0].attention
    x = rng.standard_normal((2, 150, cfg["d_model"])).astype(np.float32)
    mask = O.causal_mask(150, 150) if causal else None
    want, wc = O.attention(x, lw, cfg, osem, None, True)
    got, cache = att.forward(x, mask=mask, use_cache=True)
    assert rel_err(got, want) < TOL
    x2 = rng.standard_normal((2, 37, cfg["d_model"])).astype(np.float32)
    mask2 = O.causal_mask(37, 187) if causal else None
    want2, _ = O.attention(x2, lw, cfg, osem, wc, True)
    got2, cache2 = att.forward(x2, mask=mask2, kv_cache=cache, use_cache=True)
    assert rel_err(got2, want2) < TOL and cache2.length == 187


def test_prefill_qkv_epilogue_cache_rows(rb):
    """Prompt-sized calls in published semantics (one activation term, head_dim 128, 256 rows and more): the
    q/k/v product dequantises, rotates and appends to the cache in its read-back.  The cache rows (a direct
    function of the quantised input: rotary angles, positions, per-sequence offsets) and the attention
    output against the oracle, for a first chunk of 2 x 150 positions and a second of 2 x 140 behind it."""
    om, prompt, model = _tiny(rb, "hd128", rb.sem.BASELINE, max_seq=320, max_batch=2)
    cfg, lw = om["cfg"], om["layers"][0]
    rng = np.random.default_rng(77)
    att = model.layers[0].attention
    x = rng.standard_normal((2, 150, cfg["d_model"])).astype(np.float32)
    want, wc = O.attention(x, lw, cfg, O.BASELINE, None, True)
    got, cache = att.forward(x, mask=O.causal_mask(150, 150), use_cache=True)
    assert rel_err(cache["k"], wc["k"]) < TOL and rel_err(cache["v"], wc["v"]) < TOL
    assert rel_err(got, want) < 5e-3   # one-term int8 output projection: a flipped rounding tie moves a row
    x2 = rng.standard_normal((2, 140, cfg["d_model"])).astype(np.float32)
    want2, wc2 = O.attention(x2, lw, cfg, O.BASELINE, wc, True)
    got2, cache2 = att.forward(x2, mask=O.causal_mask(140, 290), kv_cache=cache, use_cache=True)
    assert cache2.length == 290
    assert rel_err(cache2["k"], wc2["k"]) < TOL and rel_err(cache2["v"], wc2["v"]) < TOL
    assert rel_err(got2, want2) < 5e-3


def test_wide_ffn_generation_step(rb):
    """d_ff above 8192: the down projection's prologue stages its input row in shared memory.
    Logits within tolerance and the same 32 greedy tokens as the oracle, published semantics."""
    om, prompt, model = _tiny(rb, "wide_ffn", rb.sem.BASELINE)
    osem = o_sem(rb.sem.BASELINE)
    want, _ = O.model_forward(om, prompt[None, :], osem)
    got, _ = model.forward(prompt[None, :])
    assert rel_err(got, want) < TOL
    ids = O.generate_greedy(om, prompt, G.N_NEW, osem)[len(prompt):]
    before = rb.tr.abi.lib.rotor_b200_launch_count()
    assert model.generate_greedy(prompt, G.N_NEW, use_graph=False) == ids
    per_step = (rb.tr.abi.lib.rotor_b200_launch_count() - before) / G.N_NEW
    assert per_step <= 5 * om["cfg"]["n_layers"] + 2     # the five-launch block (the unfused path takes 8 per block)
    assert model.generate_greedy(prompt, G.N_NEW, use_graph=True) == ids


@pytest.mark.parametrize("name", list(G.TINY_MODELS))
@pytest.mark.parametrize("max_seq,n_prompt", [(1100, 1040), (2100, 2040)])
def test_long_cache_generation_step(rb, name, max_seq, n_prompt):
    """Caches of 1024 and of 2048 and more positions: one-token attention keeps a slice of the cache in
    shared memory per CTA, eight slices per KV head while they fit, sixteen (a 16-CTA cluster where the
    device places one) beyond.  Last-position logits after the prompt and the next 8 greedy tokens against
    the oracle, float semantics."""
    om, _, model = _tiny(rb, name, rb.sem.REFERENCE, max_seq=max_seq)
    rng = np.random.default_rng(5150)
    prompt = rng.integers(0, om["cfg"]["vocab_size"], size=n_prompt).astype(np.int64)
    ids, steps = O.generate_greedy(om, prompt, 8, O.REFERENCE, return_logits=True)
    want = ids[len(prompt):]
    logits, cache = model.forward(prompt[None, :], use_cache=True, logits_positions="last")
    assert rel_err(logits[0, -1], steps[0]) < TOL
    nxt, _ = model.forward(np.array([[want[0]]]), past_kv_cache=cache, use_cache=True)
    assert rel_err(nxt[0, -1], steps[1]) < TOL
    assert model.generate_greedy(prompt, 8, use_graph=False) == want
    assert model.generate_greedy(prompt, 8, use_graph=True) == want


def test_empty_and_single_element_inputs(rb):
    """Zero token rows give empty outputs (the reference's NumPy path does the same); one row of one
    sequence is the smallest real call."""
    lin = rb.tr.TernaryLinear(64, 48)
    lin.load_from_int8(np.ones((48, 64), dtype=np.int8), 0.5)
    assert lin.forward(np.zeros((0, 64), dtype=np.float32)).shape == (0, 48)
    assert lin.forward(np.zeros((2, 0, 64), dtype=np.float32)).shape == (2, 0, 48)
    y = lin.forward(np.ones((1, 64), dtype=np.float32))
    assert y.shape == (1, 48) and np.allclose(y, 32.0, rtol=1e-5)
    norm = rb.tr.RMSNorm(64)
    assert norm.forward(np.zeros((0, 64), dtype=np.float32)).shape == (0, 64)
    ffn = rb.tr.GatedFFN(64, 128)
    assert ffn.gate_proj.in_features == 64
    for p in (ffn.gate_proj, ffn.up_proj, ffn.down_proj):
        p.load_from_int8(np.ones((p.out_features, p.in_features), dtype=np.int8), 0.1)
    assert ffn.forward(np.zeros((0, 64), dtype=np.float32)).shape == (0, 64)


@pytest.mark.parametrize("batch", [2, 9, 17])
def test_batched_decode_step(rb, batch):
    """One-token steps for several sequences at once against the oracle run sequence by sequence: two and more go through the
    attention that takes several sequences in one launch."""
    om, prompt, model = _tiny(rb, "hd128", rb.sem.REFERENCE, max_batch=batch)
    rng = np.random.default_rng(40 + batch)
    vocab = om["cfg"]["vocab_size"]
    ids = rng.integers(0, vocab, size=(batch, 6))
    nxt = rng.integers(0, vocab, size=(batch, 1))
    _, caches = model.forward(ids, use_cache=True)
    got, caches2 = model.forward(nxt, past_kv_cache=caches, use_cache=True)
    assert caches2[0].length == 7
    for b in range(batch):
        _, oc = O.model_forward(om, ids[b:b + 1], O.REFERENCE, use_cache=True)
        want, _ = O.model_forward(om, nxt[b:b + 1], O.REFERENCE, past_kv_cache=oc, use_cache=True)
        assert rel_err(got[b], want[0]) < TOL, (b, rel_err(got[b], want[0]))


def test_wide_ffn_many_rows(rb):
    """70 rows through an FFN whose hidden width (9216) exceeds 8192: the gating / sub-norm / quantise
    stage takes the 512-thread register-resident kernel."""
    import torch
    from rotor_b200 import ops
    d, ff, rows = 256, 9216, 70
    rng = np.random.default_rng(77)
    lw = {"gate": (O.synth_ternary(rng, ff, d), 0.02), "up": (O.synth_ternary(rng, ff, d), 0.018),
          "down": (O.synth_ternary(rng, d, ff), 0.015),
          "ffn_sub_norm": (1.0 + 0.1 * rng.standard_normal(ff)).astype(np.float32)}
    pre_w = (1.0 + 0.1 * rng.standard_normal(d)).astype(np.float32)
    x = rng.standard_normal((rows, d)).astype(np.float32)
    sem = rb.sem.REFERENCE
    ffn = rb.tr.GatedFFN(d, ff, semantics=sem)
    pre = rb.tr.RMSNorm(d, eps=sem.eps)
    pre.weight = pre_w
    ffn.ffn_norm.weight = lw["ffn_sub_norm"]
    for nm, proj in (("gate", ffn.gate_proj), ("up", ffn.up_proj), ("down", ffn.down_proj)):
        proj.load_from_int8(lw[nm][0], lw[nm][1])
    got = ffn.forward_device(ops.to_device(x, torch.float32), pre_norm=pre).cpu().numpy()
    want = O.ffn(O.rmsnorm(x, pre_w, sem.eps), lw, o_sem(sem))
    assert rel_err(got, want) < TOL, rel_err(got, want)


@pytest.mark.parametrize("ff", [4112, 6912, 7168, 7184, 8192])
def test_gated_rows_of_a_prompt(rb, ff):
    """300 rows whose gate/up product gates in its read-back: the stage that norms and quantises the float rows, at the widths
    where its thread counts change, against the same rows five at a time.  One term: a value on a tie of the quantiser may
    fall either way (one step of 1/127 of a row's largest value in a row of thousands)."""
    import torch
    ffn = rb.tr.GatedFFN(256, ff, semantics=rb.sem.BASELINE)
    g = torch.Generator(device="cuda")
    g.manual_seed(ff)
    for p in (ffn.gate_proj, ffn.up_proj, ffn.down_proj):
        p.load_from_int8(torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 0.02)
    x = torch.randn((300, 256), generator=g, device="cuda")
    got, want = ffn.forward_device(x), torch.cat([ffn.forward_device(x[i:i + 5].contiguous()) for i in range(0, 300, 5)])
    assert (got - want).norm() < 4e-3 * want.norm()
    assert ((got - want).abs().amax(1) == 0).float().mean() > 0.3   # most rows hold no tie


@pytest.mark.parametrize("batch", [3, 6])
def test_batched_greedy_generation(rb, batch):
    """Equal-length prompts generated together give, sequence by sequence, the oracle's tokens
    (three sequences: fused generation step; six: the unfused one)."""
    om, prompt, model = _tiny(rb, "hd64", rb.sem.REFERENCE, max_batch=batch)
    rng = np.random.default_rng(60 + batch)
    prompts = rng.integers(0, om["cfg"]["vocab_size"], size=(batch, 5))
    got = model.generate_greedy_batch(prompts, 12)
    assert got.shape == (batch, 12)
    for b in range(batch):
        want = O.generate_greedy(om, prompts[b], 12, O.REFERENCE)[5:]
        assert list(got[b]) == want, b
    assert np.array_equal(model.generate_greedy_batch(prompts, 12, use_graph=False), got)


@pytest.mark.parametrize("lens", [[3, 7, 5], [9, 2, 6, 4, 9, 1], [30, 17, 40], list(range(4, 21))])
def test_batched_greedy_generation_ragged(rb, lens):
    """Prompts of different lengths generated together: every sequence gives the tokens of its
    own single-prompt generation by the oracle (3 sequences: fused step; 6: unfused; 30/17/40:
    tiled prefill attention over padded rows; 17 sequences: tiled attention in the steps)."""
    import dataclasses
    batch = len(lens)
    sem, osem = dataclasses.replace(rb.sem.REFERENCE, causal=True), dataclasses.replace(O.REFERENCE, causal=True)
    om, prompt, model = _tiny(rb, "hd64", sem, max_batch=batch)
    rng = np.random.default_rng(70 + batch + lens[0])
    prompts = [rng.integers(0, om["cfg"]["vocab_size"], size=n) for n in lens]
    new = 8
    got = model.generate_greedy_batch(prompts, new)
    assert got.shape == (batch, new)
    for b in range(batch):
        want = O.generate_greedy(om, prompts[b], new, osem)[lens[b]:]
        assert list(got[b]) == want, b
    assert np.array_equal(model.generate_greedy_batch(prompts, new, use_graph=False), got)
    with pytest.raises(ValueError):  # without a causal mask a row would attend to its padding
        _tiny(rb, "hd64", rb.sem.REFERENCE, max_batch=batch)[2].generate_greedy_batch(prompts, new)


@pytest.mark.parametrize("shape", [(1024, 8, 2, 1536), (2560, 20, 5, 6912), (8192, 64, 8, 9216), (512, 8, 8, 512), (512, 4, 2, 512),
                                   (768, 12, 4, 512), (1280, 20, 4, 512), (768, 6, 1, 512), (1792, 14, 2, 512), (1024, 16, 2, 512)])
@pytest.mark.parametrize("batch,context", [(2, 129), (3, 30), (4, 300), (5, 300), (16, 30), (33, 129)])
def test_batched_steps_equal_single_sequences(rb, shape, batch, context):
    """Two steps of several sequences (row stages with few rows, merged runs of the decode attention, sums cleared ahead
    of split products) against the same steps of each sequence alone: widths of every thread count, contexts with and
    without several runs per sequence, ragged runs, one to eight query heads per key head.  Three activation terms: float32 rounding is all that may differ."""
    import torch
    d, heads, kv, ff = shape
    cfg = dict(vocab_size=512, d_model=d, n_layers=2, n_heads=heads, n_kv_heads=kv, d_ff=ff)
    model = rb.synth.random_model_on_device(cfg, seed=batch + context, semantics=rb.sem.REFERENCE, max_seq=context + 2, max_batch=batch,
                                            max_rows=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(d + batch)
    held = []
    for layer in model.layers:
        held.append([torch.randn((batch, kv, context, d // heads), generator=g, device="cuda") for _ in range(2)])
    ids = np.random.default_rng(batch).integers(0, 512, size=(2, batch, 1))

    def steps(rows):
        for layer, (k, v) in zip(model.layers, held):
            for cache, t in zip(layer.attention.ensure_cache(batch, context + 2), (k, v)):
                cache[:len(rows), :, :context] = t[rows]
        caches = [rb.tr.KVCache(layer.attention, context, len(rows)) for layer in model.layers]
        out = []
        for i in range(2):
            logits, caches = model.forward_last_logits_device(ids[i][rows], caches)
            out.append(logits.clone())
        return torch.stack(out, 1)

    got = steps(list(range(batch)))
    for b in (0, batch // 2, batch - 1):
        assert rel_err(got[b].cpu().numpy(), steps([b])[0].cpu().numpy()) < 2e-4, b   # about 60 float32 sums of up to 9216 in a row


@pytest.mark.parametrize("heads,kv,batch,context,capacity", [(4, 1, 5, 0, 4), (4, 1, 7, 3, 5), (8, 2, 20, 37, 39), (12, 4, 16, 41, 43),
                                                            (8, 1, 17, 26, 28), (20, 5, 8, 47, 49), (20, 5, 8, 6, 700), (20, 5, 24, 9, 11),
                                                            (16, 2, 64, 21, 23), (8, 8, 40, 19, 1500), (16, 8, 90, 11, 300),
                                                            (32, 4, 8, 333, 335), (20, 4, 35, 150, 152), (8, 8, 37, 65, 67), (16, 2, 150, 97, 600)])
def test_runs_of_batched_steps(rb, heads, kv, batch, context, capacity):
    """Steps whose sequences are cut into every number of runs that the rule gives, with empty runs, rings that wrap, runs that
    are no multiple of a warp's keys and outputs that do not divide by the runs, against each sequence alone.  Two steps: the
    second reads the row that the first appended.  Three activation terms: float32 rounding is all that may differ."""
    import torch
    cfg = dict(vocab_size=512, d_model=heads * (128 if heads in (20, 32) else 64), n_layers=1, n_heads=heads, n_kv_heads=kv, d_ff=512)
    model = rb.synth.random_model_on_device(cfg, seed=batch, semantics=rb.sem.REFERENCE, max_seq=capacity, max_batch=batch, max_rows=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(heads + batch)
    held = [torch.randn((batch, kv, context, cfg["d_model"] // heads), generator=g, device="cuda") for _ in range(2)]
    ids = np.random.default_rng(batch).integers(0, 512, size=(2, batch, 1))

    def steps(rows):
        at = model.layers[0].attention
        for cache, t in zip(at.ensure_cache(batch, capacity), held):
            cache[:len(rows), :, :context] = t[rows]
        caches, out = [rb.tr.KVCache(at, context, len(rows))], []
        for i in range(2):
            logits, caches = model.forward_last_logits_device(ids[i][rows], caches)
            out.append(logits.clone())
        return torch.stack(out, 1)

    got = steps(list(range(batch)))
    for b in (0, batch - 1):
        assert rel_err(got[b].cpu().numpy(), steps([b])[0].cpu().numpy()) < 2e-4, b


@pytest.mark.parametrize("heads,kv", [(4, 2), (8, 1), (3, 3)])
@pytest.mark.parametrize("batch,context,hidden", [(5, 300, 4), (5, 300, 45), (5, 300, 300), (16, 30, 17), (33, 129, 128), (18, 5, 5)])
def test_infinite_scores_weigh_nothing(rb, heads, kv, batch, context, hidden):
    """Cached keys whose score is minus infinity, the first `hidden` of a context, in steps of several sequences: a warp's
    first keys, whole runs, everything but the new key.  The same as keys so far below the others that their weight
    underflows to zero, to the bit."""
    import torch
    d = 64 * heads
    at = rb.tr.MultiHeadAttention(d, heads, kv, semantics=rb.sem.REFERENCE, max_seq=context + 1, max_batch=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(context + hidden + heads)
    for p in (at.k_proj, at.v_proj, at.o_proj):
        p.load_from_int8(torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 0.05)
    at.q_proj.load_from_int8(torch.ones((d, d), device="cuda", dtype=torch.int8), 0.1 / d)   # positive rows: positive queries
    x = np.random.default_rng(batch).uniform(0.5, 1.5, size=(batch, 1, d)).astype(np.float32)
    k, v = at.ensure_cache()
    v[:, :, :context] = torch.randn(v[:, :, :context].shape, generator=g, device="cuda")
    keys = torch.randn(k[:, :, :context].shape, generator=g, device="cuda")
    got = []
    for low in (-np.inf, -1e30):
        k[:, :, :context] = keys
        k[:, :, :hidden, 5] = low
        got.append(at.forward(x, kv_cache=rb.tr.KVCache(at, context, batch))[0])
    assert np.isfinite(got[1]).all() and np.abs(got[1]).max() > 0
    assert np.array_equal(*got)


def _attention_layer(rb, d, heads, kv, seed, **kw):
    """An attention layer with random weights, and the weights (times their scales) in float64."""
    import torch
    at = rb.tr.MultiHeadAttention(d, heads, kv, **kw)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    mats = []
    for p in (at.q_proj, at.k_proj, at.v_proj, at.o_proj):
        w = torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8)
        p.load_from_int8(w, 0.04)
        mats.append(w.double() * float(np.float32(0.04)))
    return at, mats


@pytest.mark.parametrize("heads,kv,batch,seq", [(3, 1, 3, 100), (4, 1, 2, 131), (5, 5, 1, 300)])
def test_qkv_rows_of_a_prompt(rb, heads, kv, batch, seq):
    """256 rows and more of one activation term: the q/k/v product finishes its rows in its read-back (an odd number of heads, tiles
    across sequences, a cache that holds something already).  The cache against the one that portions below 16 tokens
    leave (float32 rounding), the outputs within what a quantiser's ties explain."""
    sem = rb.sem.BASELINE
    at, _ = _attention_layer(rb, 128 * heads, heads, kv, heads + seq, semantics=sem, max_seq=seq + 7, max_batch=batch)
    x = np.random.default_rng(seq).standard_normal((batch, seq + 7, 128 * heads)).astype(np.float32)

    def run(cuts):
        out, cache = [], None
        for a, b in zip(cuts, cuts[1:]):
            y, cache = at.forward(x[:, a:b], kv_cache=cache, use_cache=True)
            out.append(y)
        return np.concatenate(out, 1), cache["k"], cache["v"]

    whole, k, v = run([0, 7, seq + 7])
    parts, k2, v2 = run(list(range(0, seq + 7, 15)) + [seq + 7])
    assert rel_err(k, k2) < 1e-6 and rel_err(v, v2) < 1e-6
    assert np.linalg.norm(whole - parts) < 2e-2 * np.linalg.norm(parts)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("heads,kv,batch,past,seq", [(1, 1, 1, 0, 16), (2, 1, 1, 0, 65), (4, 1, 3, 300, 33), (8, 1, 2, 64, 47), (5, 5, 2, 10, 300),
                                                     (16, 4, 9, 0, 200), (3, 3, 5, 130, 1300)])
def test_prompt_attention_against_float64(rb, heads, kv, batch, past, seq, causal):
    """Prompts behind cached rows whose scores rise and fall by far more than the weights' reference follows without moving, more
    query tiles than SMs (each CTA several, of unequal length), tiles of one and two key tiles, rows that see nothing of a
    tile, a last tile without whole rows.  Three activation terms."""
    import dataclasses
    import torch
    d = 128 * heads
    sem = dataclasses.replace(rb.sem.REFERENCE, causal=causal)
    at, (wq, wk, wv, wo) = _attention_layer(rb, d, heads, kv, heads + seq + past, semantics=sem, max_seq=past + seq, max_batch=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(seq)
    x = torch.randn((batch, seq, d), generator=g, device="cuda")
    k, v = at.ensure_cache()
    if past:
        k[:, :, :past] = torch.randn(k[:, :, :past].shape, generator=g, device="cuda") * (torch.arange(past, device="cuda") % 97 / 8.0)[:, None]
        v[:, :, :past] = torch.randn(v[:, :, :past].shape, generator=g, device="cuda")
    held = [t[:, :, :past].double() for t in (k, v)]
    cache = rb.tr.KVCache(at, past, batch) if past else None
    got = torch.as_tensor(at.forward(x.cpu().numpy(), kv_cache=cache)[0]).cuda().double()
    rows = x.double()
    q, kn, vn = ((rows @ w.T).reshape(batch, seq, -1, 128).transpose(1, 2) for w in (wq, wk, wv))
    kk, vv = (torch.cat(t, 2).repeat_interleave(heads // kv, 1) for t in zip(held, (kn, vn)))
    want, top = torch.empty_like(rows), 0.0
    for b in range(batch):
        s = q[b] @ kk[b].transpose(-1, -2) * 128 ** -0.5
        top = max(top, float(s.abs().max()))
        if causal:
            at_, key = torch.arange(seq, device="cuda")[:, None] + past, torch.arange(past + seq, device="cuda")[None]
            s = s.masked_fill(key > at_, -np.inf)
        want[b] = (s.softmax(-1) @ vv[b]).transpose(0, 1).reshape(seq, d) @ wo.T
    want = want / (want.square().mean(-1, keepdim=True) + sem.eps).sqrt()
    # an operand keeps 16 bits: a score of size s is off by up to 2^-16 s, its weight by as much of itself
    assert (got - want).norm() < (3e-5 + top * 2.0 ** -16) * want.norm(), float((got - want).norm() / want.norm())


@pytest.mark.parametrize("rows", [2, 4, 5, 9])
@pytest.mark.parametrize("ff", [10880, 10944])
def test_ffn_sums_cleared_by_stage_or_memset(rb, ff, rows):
    """Three terms, at the width where a row's gate and up sums pass the size that a stage clears itself, in the stages of few
    and of more rows, against the rows one at a time (float32 rounding is all that may differ)."""
    import torch
    ffn = rb.tr.GatedFFN(512, ff, semantics=rb.sem.REFERENCE)
    g = torch.Generator(device="cuda")
    g.manual_seed(ff + rows)
    for p in (ffn.gate_proj, ffn.up_proj, ffn.down_proj):
        p.load_from_int8(torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 0.02)
    x = torch.randn((rows, 512), generator=g, device="cuda")
    got, want = ffn.forward_device(x), torch.cat([ffn.forward_device(x[i:i + 1].contiguous()) for i in range(rows)])
    assert (got - want).norm() < 2e-5 * want.norm()


@pytest.mark.parametrize("terms,few,many", [(1, (5, 8, 9), (10, 16)), (3, (3,), (4, 5))])
def test_ffn_rows_that_the_down_product_finishes(rb, terms, few, many):
    """Up to nine columns of 6912 the down product leaves finished rows, one launch less than with its sums in memory.  The same stages
    and the same integer sums: one term's rows are equal to the bit, three terms' sums may be rounded once more each."""
    import torch
    lib, sem = rb.tr.abi.lib, {1: rb.sem.BASELINE, 3: rb.sem.REFERENCE}[terms]
    ffn = rb.tr.GatedFFN(2560, 6912, semantics=sem)
    g = torch.Generator(device="cuda")
    g.manual_seed(terms)
    for p in (ffn.gate_proj, ffn.up_proj, ffn.down_proj):
        p.load_from_int8(torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 0.02)
    x = torch.randn((max(many), 2560), generator=g, device="cuda")

    def run(rows):
        before = lib.rotor_b200_launch_count()
        y = ffn.forward_device(x[:rows])
        return y, lib.rotor_b200_launch_count() - before

    sums = [run(rows) for rows in many]
    for rows in few:
        y, launches = run(rows)
        assert launches == sums[0][1] - 1, rows
        for want, _ in sums:
            n = min(rows, len(want))
            assert torch.equal(y[:n], want[:n]) if terms == 1 else (y[:n] - want[:n]).norm() < 1e-6 * want[:n].norm(), rows
    rb.tr.abi.device_status()


@pytest.mark.parametrize("d", [512, 1536, 2560])
def test_prompt_rows_of_many_equal_few(rb, d):
    """2300 rows of a prompt of two sequences (three rounds of six CTAs an SM in the residual stages, four of five) against the
    1150 of each sequence alone (two rounds either way: five CTAs; rows of 2560 with three terms: always five).  The integer sums are the same and the stages add in the same order."""
    import torch
    model = rb.synth.random_model_on_device(dict(vocab_size=512, d_model=d, n_layers=2, n_heads=d // 128, n_kv_heads=1, d_ff=512), seed=d,
                                            semantics=rb.sem.REFERENCE, max_seq=1150, max_batch=2, max_rows=2300)
    ids = np.random.default_rng(d).integers(0, 512, size=(2, 1150))
    got = model.forward_last_logits_device(ids)[0].clone()
    for b in range(2):
        want = model.forward_last_logits_device(ids[b:b + 1])[0]
        assert rel_err(got[b].cpu().numpy(), want[0].cpu().numpy()) < 1e-5, b


def _off(t):
    """The same values, four bytes behind a 16-byte boundary."""
    import torch
    return torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 300])
def test_rmsnorm_off_a_16_byte_boundary(rb, rows):
    """Rows, weights and results that start at any float: the register stage moves four at a time and leaves these to the other."""
    import torch
    abi, n = rb.tr.abi, 2560
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    x, w = torch.randn((rows, n), generator=g, device="cuda"), torch.rand(n, generator=g, device="cuda")
    want = x.double() / (x.double().square().mean(-1, keepdim=True) + 1e-6).sqrt() * w.double()
    for which in range(8):
        a, b, y = (_off(t) if which >> i & 1 else t.clone() for i, t in enumerate((x, w, torch.empty_like(x))))
        abi.check(abi.lib.rotor_b200_rmsnorm(abi.ptr(a), rows, n, abi.ptr(b), 1e-6, abi.ptr(y), abi.stream()))
        abi.device_status()
        assert (y.double() - want).norm() < 1e-6 * want.norm(), which   # a few float32 roundings


@pytest.mark.parametrize("batch,seq", [(1, 1), (2, 1), (4, 1), (1, 3), (5, 1), (1, 300)])
def test_attention_rows_off_a_16_byte_boundary(rb, batch, seq):
    """Rows in, rows out and the sub-norm's weights at any float, against the same rows on a boundary.  Three activation terms: other
    stages round float32 sums of 256 in another order, and a term's quantiser moves by that."""
    import ctypes as C
    import torch
    abi, d = rb.tr.abi, 256
    at, _ = _attention_layer(rb, d, 4, 2, batch + seq, semantics=rb.sem.REFERENCE, max_seq=seq, max_batch=batch)
    at.attn_norm.weight = (1 + 0.1 * np.random.default_rng(seq).standard_normal(d)).astype(np.float32)
    g = torch.Generator(device="cuda")
    g.manual_seed(seq)
    x = torch.randn((batch * seq, d), generator=g, device="cuda")
    cfg, lw = at._cfg_struct(at.semantics, batch, seq, batch * seq), abi.LayerWeights()
    at.fill_layer_struct(lw)
    ws, norm, out = at._workspace_for(cfg, batch * seq), at.attn_norm.device_weight(), []
    for place in (torch.clone, _off):
        a, w, y = place(x), place(norm), place(torch.empty_like(x))
        lw.attn_sub_norm = abi.ptr(w)
        abi.check(abi.lib.rotor_b200_attention_forward(C.byref(cfg), C.byref(lw), abi.ptr(a), batch, seq, 0, abi.ptr(y), abi.ptr(ws), ws.numel(),
                                                       abi.stream()))
        abi.device_status()
        out.append(y.double())
    assert (out[1] - out[0]).norm() < 1e-5 * out[0].norm()


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 9, 300])
def test_ffn_rows_off_a_16_byte_boundary(rb, rows):
    """The same of the feed-forward, whose row norm and sub-norm may start anywhere too.  One and two rows on a boundary are two launches
    whose prologues move four floats at a time; off it they go through the stages."""
    import torch
    d, ff = 512, 1536
    ffn, pre = rb.tr.GatedFFN(d, ff, semantics=rb.sem.REFERENCE), rb.tr.RMSNorm(d)
    g = torch.Generator(device="cuda")
    g.manual_seed(rows)
    for p in (ffn.gate_proj, ffn.up_proj, ffn.down_proj):
        p.load_from_int8(torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 0.02)
    norms = [torch.rand(n, generator=g, device="cuda") + 0.5 for n in (d, ff)]
    x = torch.randn((rows, d), generator=g, device="cuda")
    out = []
    for place in (torch.clone, _off):
        for norm, w in zip((pre, ffn.ffn_norm), norms):
            held = place(w)
            norm.device_weight = lambda held=held: held
        out.append(ffn.forward_device(place(x), pre_norm=pre).double())
        rb.tr.abi.device_status()
    assert (out[1] - out[0]).norm() < 1e-5 * out[0].norm()


@pytest.mark.parametrize("seq", [33, 391, 700])
def test_prompt_rows_do_not_depend_on_earlier_calls(rb, seq):
    """A prompt whose last query tile has rows past its end, behind calls of other magnitudes: what shared memory still holds of those
    lies in these rows, and must not change what the others round to."""
    import dataclasses
    at, _ = _attention_layer(rb, 512, 4, 1, 5, semantics=dataclasses.replace(rb.sem.REFERENCE, causal=True), max_seq=1024)
    x = np.random.default_rng(seq).standard_normal((1, 1024, 512)).astype(np.float32)
    got = []
    for scale in (0.0, 0.01, 3.0, 30.0, 300.0):
        at.forward(x * np.float32(scale))
        got.append(at.forward(x[:, :seq])[0])
    assert all(np.array_equal(got[0], y) for y in got[1:])


@pytest.mark.parametrize("heads,kv,batch,context", [(20, 5, 64, 1500), (8, 8, 40, 1900), (20, 5, 56, 1900)])
def test_long_contexts_are_summed_in_parts(rb, heads, kv, batch, context):
    """Steps in which a warp adds up hundreds of keys are no further from float64 than the same sequences eight at a time, each cut into
    runs of short sums.  (Quantisers make up most of either error.  The ratio was seen at 0.99 to 1.02; sums of a whole
    share in a row make it 1.05 to 1.14.)"""
    import ctypes as C
    import torch
    abi, d, dim = rb.tr.abi, 128 * heads, 128
    at, (wq, wk, wv, wo) = _attention_layer(rb, d, heads, kv, batch, semantics=rb.sem.REFERENCE, max_seq=context + 1, max_batch=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(context)
    held = [torch.randn((batch, kv, context, dim), generator=g, device="cuda") for _ in range(2)]
    x = torch.randn((batch, d), generator=g, device="cuda") * (0.5 / 0.04 / d ** 0.5)   # scores of the size that a model has

    def run(rows):
        n = len(x[rows])
        for cache, t in zip(at.ensure_cache(), held):
            cache[:n, :, :context] = t[rows]
        cfg, lw, y = at._cfg_struct(at.semantics, batch, context + 1, n), abi.LayerWeights(), torch.empty_like(x[rows])
        at.fill_layer_struct(lw)
        ws = at._workspace_for(cfg, n)
        abi.check(abi.lib.rotor_b200_attention_forward(C.byref(cfg), C.byref(lw), abi.ptr(x[rows].contiguous()), n, 1, context, abi.ptr(y),
                                                       abi.ptr(ws), ws.numel(), abi.stream()))
        abi.device_status()
        return y.double()

    q, kn, vn = ((x.double() @ w.T).view(batch, -1, 1, dim) for w in (wq, wk, wv))
    k, v = (torch.cat((t.double(), n), 2) for t, n in zip(held, (kn, vn)))
    scores = torch.einsum("bkgd,bktd->bkgt", q.view(batch, kv, heads // kv, dim), k) * dim ** -0.5
    want = torch.einsum("bkgt,bktd->bkgd", scores.softmax(-1), v).reshape(batch, d) @ wo.T
    want = want / (want.square().mean(-1, keepdim=True) + at.semantics.eps).sqrt()
    few = torch.cat([run(slice(i, i + 8)) for i in range(0, batch, 8)])
    assert (run(slice(0, batch)) - want).norm() < 1.04 * (few - want).norm()


@pytest.mark.parametrize("heads,kv,batch,past,seq", [(20, 5, 2, 0, 700), (4, 1, 3, 300, 33), (8, 8, 1, 0, 1300), (20, 5, 8, 0, 128)])
def test_prompt_attention_keeps_its_operand_bits(rb, heads, kv, batch, past, seq):
    """The error of an attention layer over a prompt, which the 16-bit operands of the tensor cores make up: seen at 5.6e-6 to 6.6e-6,
    and at 6.7e-6 to 8.0e-6 with scores of three products."""
    import dataclasses
    import torch
    d = 128 * heads
    sem = dataclasses.replace(rb.sem.REFERENCE, causal=True)
    at, _ = _attention_layer(rb, d, heads, kv, seq, semantics=sem, max_seq=past + seq, max_batch=batch)
    g = torch.Generator(device="cuda")
    g.manual_seed(seq)
    mats = []
    for p in (at.q_proj, at.k_proj, at.v_proj, at.o_proj):
        w, scale = torch.randint(-1, 2, (p.out_features, p.in_features), generator=g, device="cuda", dtype=torch.int8), 1.633 * d ** -0.5
        p.load_from_int8(w, scale)
        mats.append(w.double() * float(np.float32(scale)))
    held = [torch.randn((batch, kv, past, 128), generator=g, device="cuda") for _ in range(2)]
    for cache, t in zip(at.ensure_cache(), held):
        cache[:, :, :past] = t
    x = torch.randn((batch, seq, d), generator=g, device="cuda")
    got = torch.as_tensor(at.forward(x.cpu().numpy(), kv_cache=rb.tr.KVCache(at, past, batch) if past else None)[0]).cuda().double()
    q, kn, vn = ((x.double() @ w.T).reshape(batch, seq, -1, 128).transpose(1, 2) for w in mats[:3])
    k, v = (torch.cat((t.double(), n), 2).repeat_interleave(heads // kv, 1) for t, n in zip(held, (kn, vn)))
    hidden = torch.arange(past + seq, device="cuda")[None] > torch.arange(seq, device="cuda")[:, None] + past
    want = torch.stack([((q[b] @ k[b].transpose(-1, -2) * 128 ** -0.5).masked_fill(hidden, -np.inf).softmax(-1) @ v[b]).transpose(0, 1).reshape(seq, d)
                        @ mats[3].T for b in range(batch)])
    want = want / (want.square().mean(-1, keepdim=True) + sem.eps).sqrt()
    assert (got - want).norm() < (6.2e-6 if seq == 128 else 6.6e-6 if seq == 33 else 7e-6) * want.norm(), float((got - want).norm() / want.norm())
