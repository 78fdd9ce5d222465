"""GPU: the many-row LM head at the edges of its tiles (token rows 16 / 32 / 64 / 128 per pass, vocabulary shares in units of
16 rows, tiles of 256) against a float64 product of the same hidden rows, and its greedy pick."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[139, 4099], ids=lambda v: f"vocab{v}")
def model(request):
    import torch
    from rotor_b200.synth import random_model_on_device
    m = random_model_on_device(dict(vocab_size=request.param, d_model=256, n_layers=1, n_heads=2, n_kv_heads=1, d_ff=512), seed=3,
                               max_seq=300, max_batch=48)
    e = m._embed
    e[request.param // 2:request.param // 2 + 40] = e[3:43]     # equal rows far apart: the lower index has to win
    torch.cuda.synchronize()
    return m


@pytest.mark.parametrize("rows", [5, 16, 17, 32, 33, 64, 65, 128, 129, 257])
def test_logits(model, rows):
    ids = np.random.default_rng(rows).integers(0, model.vocab_size, size=(1, rows))
    hidden, _ = model.forward(ids, return_logits=False)
    logits, _ = model.forward(ids)
    want = hidden[0].astype(np.float64) @ model.embed_tokens.astype(np.float64).T
    # hi + lo keep 16 bits of a hidden value, sums are float32: 2^-17 and about 2^-21 of the terms' root sum of squares
    err = np.linalg.norm(logits[0] - want) / np.linalg.norm(want)
    assert err < 2.0 ** -16, err


@pytest.mark.parametrize("batch", [5, 16, 17, 33, 48])
def test_pick(model, batch):
    ids = np.random.default_rng(batch).integers(0, model.vocab_size, size=(batch, 5))
    logits, _ = model.forward(ids, logits_positions="last")
    first = model.generate_greedy_batch(ids, 1)[:, 0]
    assert np.array_equal(first, logits[:, 0].argmax(-1))
    assert (first < model.vocab_size // 2).any()
