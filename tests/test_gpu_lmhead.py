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


@pytest.fixture(scope="module")
def tall():
    """A vocabulary of several 256-row tiles per CTA, the last ragged, and a table of several rings of stages per tile."""
    from rotor_b200.synth import random_model_on_device
    return random_model_on_device(dict(vocab_size=148 * 600 + 5, d_model=512, n_layers=1, n_heads=4, n_kv_heads=1, d_ff=512), seed=5,
                                  max_seq=300, max_batch=129, max_rows=390)


@pytest.mark.parametrize("rows", [5, 16, 17, 33, 65, 129])
def test_logits_of_several_tiles(tall, rows):
    import torch
    ids = np.random.default_rng(rows).integers(0, tall.vocab_size, size=(1, rows))
    hidden, _ = tall.forward(ids, return_logits=False)
    logits, _ = tall.forward(ids)
    want = (torch.from_numpy(hidden[0]).cuda().double() @ tall._embed.double().T).cpu().numpy()
    err = np.linalg.norm(logits[0] - want) / np.linalg.norm(want)
    assert err < 2.0 ** -16, err
    assert np.abs(logits[0] - want).max() < 2.0 ** -12 * np.abs(want).max()     # (no tile missing: one wrong row would show)


@pytest.mark.parametrize("batch", [5, 17, 33, 65, 129])
def test_pick_of_equal_rows(tall, batch):
    """Every sequence's best vocabulary row twice, the second in the next lane, another half of the tile, the next tile, the
    ragged last tile, another CTA: the lower index is picked."""
    import torch
    ids = np.stack(divmod(np.random.default_rng(batch).permutation(10000)[:batch], 100), 1)     # (no two alike)
    hidden, _ = tall.forward(ids, return_logits=False)
    h = torch.from_numpy(hidden[:, -1]).cuda()
    units, parts = (tall.vocab_size + 15) // 16, min((tall.vocab_size + 127) // 128, torch.cuda.get_device_properties(0).multi_processor_count)
    kept, first = tall._embed.clone(), []
    try:
        for b in range(batch):
            cta = 1 + (b * 37) % (parts - 9)
            at = units * cta // parts * 16 + b // 5
            far = [1, 130, 256, 520, (units * (cta + 7) // parts - units * cta // parts) * 16 + 3][b % 5]
            first.append(at)
            tall._embed[at] = tall._embed[at + far] = (4 * h[b]).to(torch.bfloat16)
        assert len(set(first)) == batch
        got = tall.generate_greedy_batch(ids, 1)[:, 0]
        logits, _ = tall.forward(ids, logits_positions="last")
    finally:
        tall._embed.copy_(kept)
    assert np.array_equal(logits[:, 0].argmax(-1), first)
    assert np.array_equal(got, first)
