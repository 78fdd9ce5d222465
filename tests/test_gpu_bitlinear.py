"""GPU: activation quantiser (a13) and BitLinear (a5/a14) through the C ABI.
Integer results are compared bit-for-bit; float32 outputs within 1e-3 of the output RMS
(max-abs), the tolerance stated for this path."""
import os

import numpy as np
import pytest

import golden_inputs as G
from oracle import bitlinear_np as O

pytestmark = pytest.mark.gpu
TOL = 1e-3  # max-abs error relative to the output RMS


def rel_err(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.max(np.abs(a - b)) / np.sqrt(np.mean(b ** 2)))


@pytest.fixture(scope="module")
def ops():
    from rotor_b200 import ops
    return ops


@pytest.fixture(scope="module")
def abi():
    from rotor_b200 import abi
    return abi


@pytest.mark.parametrize("terms", [1, 2, 3])
def test_quantize_rows_bit_exact(ops, golden_dir, terms):
    x = G.quant_inputs()
    xq, sx, xsum = ops.quantize_rows(x, terms)
    q, s = O.quantize_rows(x, terms)
    m, k = x.shape
    got = xq.cpu().numpy().reshape(m, terms, -1)
    assert np.array_equal(got[:, :, :k], q)
    assert not got[:, :, k:].any()
    assert np.array_equal(sx.cpu().numpy().reshape(m, terms), s)
    assert np.array_equal(xsum.cpu().numpy().reshape(m, terms), q.astype(np.int32).sum(axis=2))
    if terms == 1:
        z = np.load(os.path.join(golden_dir, "quantize.npz"))
        assert np.array_equal(got[:, 0, :k], z["q"]) and np.array_equal(sx.cpu().numpy(), z["s"])


@pytest.mark.parametrize("k", [8, 72, 2560, 6912, 28672])
def test_quantize_rows_sizes(ops, k):
    rng = np.random.default_rng(k)
    x = (rng.standard_normal((2, k)) * 3).astype(np.float32)
    xq, sx, xsum = ops.quantize_rows(x, 2)
    q, s = O.quantize_rows(x, 2)
    assert np.array_equal(xq.cpu().numpy().reshape(2, 2, -1)[:, :, :k], q)
    assert np.array_equal(sx.cpu().numpy().reshape(2, 2), s)


@pytest.mark.parametrize("variant", ["dp4a", "mma"])
@pytest.mark.parametrize("shape", [(16, 128, 1), (20, 72, 3), (6912, 2560, 1), (6912, 2560, 3), (2560, 6912, 2),
                                   (640, 2560, 1), (48, 1280, 8), (33, 260, 11)])
def test_integer_accumulators_bit_exact(ops, abi, variant, shape):
    out, inn, ncols = shape
    rng = np.random.default_rng(out + inn + ncols)
    w = O.synth_ternary(rng, out, inn)
    tiles = ops.int8_to_tiles(w)
    kpad = abi.lib.rotor_b200_in_padded(inn)
    q = np.zeros((ncols, kpad), dtype=np.int8)
    q[:, :inn] = rng.integers(-128, 128, size=(ncols, inn), dtype=np.int8)   # full int8 range incl. -128
    xq = ops.to_device(q)
    xsum = ops.to_device(q.astype(np.int32).sum(axis=1).astype(np.int32))
    v = abi.VARIANT_DP4A if variant == "dp4a" else abi.VARIANT_MMA
    acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, v).cpu().numpy()
    want = q[:, :inn].astype(np.int32) @ w.astype(np.int32).T
    assert np.array_equal(acc, want)
    abi.device_status()


@pytest.mark.parametrize("shape", [(6912, 2560, 130), (2560, 6912, 257), (48, 1280, 32), (33, 260, 300), (640, 2560, 1024),
                                   (400, 2560, 517), (3840, 384, 256), (272, 128, 700), (2560, 2560, 64), (528, 640, 100),
                                   (6912, 2560, 192)])
def test_many_column_product_bit_exact(ops, abi, shape):
    """Prefill-sized products (32 activation columns and more) take the tcgen05 kernel (TMA-fed token
    operand, weights decoded into shared memory, int32 accumulators in tensor memory); the mma.sync
    tiled GEMM remains behind ROTOR_B200_NO_TCGEN05.  Ragged token counts, row counts that do not fill
    the 256-row tile, and K that is not a multiple of the 128-wide weight tile."""
    out, inn, ncols = shape
    rng = np.random.default_rng(out * 3 + inn + ncols)
    w = O.synth_ternary(rng, out, inn)
    tiles = ops.int8_to_tiles(w)
    kpad = abi.lib.rotor_b200_in_padded(inn)
    q = np.zeros((ncols, kpad), dtype=np.int8)
    q[:, :inn] = rng.integers(-128, 128, size=(ncols, inn), dtype=np.int8)
    xq = ops.to_device(q)
    xsum = ops.to_device(q.astype(np.int32).sum(axis=1).astype(np.int32))
    acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, abi.VARIANT_AUTO).cpu().numpy()
    want = q[:, :inn].astype(np.int32) @ w.astype(np.int32).T
    assert np.array_equal(acc, want)
    # the column-chunked tensor-core GEMV gives the same integers
    acc2 = ops.bitlinear_acc(tiles, out, inn, xq, xsum, abi.VARIANT_MMA).cpu().numpy()
    assert np.array_equal(acc2, want)


@pytest.mark.parametrize("shape", [(18939, 100, 129), (9473, 260, 300), (6403, 384, 700), (2560, 6912, 4100), (19000, 1024, 255), (37888, 128, 130)])
def test_tiles_of_cta_pairs_bit_exact(ops, abi, shape):
    """Products with a 256 x 256 tile for every pair of SMs: one to 54 K steps a tile (fewer than the decoders look ahead),
    a second half of a tile without tokens, rows and tokens that fill no tile, several tiles a pair."""
    import torch
    out, inn, ncols = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(out + ncols)
    w = torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8)
    q = torch.zeros((ncols, abi.lib.rotor_b200_in_padded(inn)), device="cuda", dtype=torch.int8)
    q[:, :inn] = torch.randint(-128, 128, (ncols, inn), generator=g, device="cuda", dtype=torch.int8)
    acc = ops.bitlinear_acc(ops.int8_to_tiles(w), out, inn, q, q.sum(1, dtype=torch.int32), abi.VARIANT_AUTO)
    assert torch.equal(acc.double(), q[:, :inn].double() @ w.double().T)
    abi.device_status()


@pytest.mark.parametrize("terms", [1, 2, 3])
@pytest.mark.parametrize("shape", [(1, 4), (17, 132), (3001, 1924), (2560, 8192), (640, 9220), (8192, 2048)])
@pytest.mark.parametrize("rows", [1, 2, 4, 5])
def test_layer_call_of_few_rows(ops, abi, shape, rows, terms):
    """One launch up to four rows of six columns, quantiser, product and dequantiser above: both against the general path
    (the variant forced), with a row of zeros, NaN and infinities, rows that start off a 16-byte boundary, and y on x."""
    import torch
    out, inn = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(out + inn + rows + terms)
    tiles = ops.int8_to_tiles(torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8))
    buf = torch.randn(rows * inn + 1, generator=g, device="cuda")
    buf[:2 * inn:2] *= 1e-3
    for x in (buf[:-1].view(rows, inn), buf[1:].view(rows, inn)):
        for spoil in (None, 0.0, float("nan"), float("inf")):
            x = x.clone() if x.data_ptr() % 16 == 0 else x
            if spoil == 0.0:
                x[rows - 1] = 0.0
            elif spoil is not None:
                x[rows - 1, inn // 2] = spoil
            got = ops.bitlinear_forward(tiles, out, inn, x, terms, 0.037)
            want = ops.bitlinear_forward(tiles, out, inn, x, terms, 0.037, variant=abi.VARIANT_MMA)
            if terms == 1:
                assert torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)) and torch.equal(got.isnan(), want.isnan())
            else:  # the terms' sum may be fused: one rounding of the largest term
                fin = want.isfinite()
                assert torch.equal(got.isfinite(), fin)
                scale = want[fin].abs().max() if fin.any() else torch.ones((), device="cuda")
                assert (got[fin] - want[fin]).abs().max().nan_to_num(0.0) <= 3e-7 * scale if fin.any() else True
    if out <= inn:
        x = torch.randn((rows, inn), generator=g, device="cuda")
        want = ops.bitlinear_forward(tiles, out, inn, x, terms, 0.5, variant=abi.VARIANT_MMA)
        ws = torch.empty(abi.lib.rotor_b200_bitlinear_workspace_bytes(out, inn, rows, terms), dtype=torch.uint8, device="cuda")
        abi.check(abi.lib.rotor_b200_bitlinear_forward(abi.ptr(tiles), out, inn, abi.ptr(x), rows, terms, 0.5, None, abi.ptr(x),
                                                       abi.ptr(ws), ws.numel(), 0, abi.stream()))
        got = x.flatten()[:rows * out].view(rows, out)
        assert (got - want).abs().max() <= 3e-7 * want.abs().max()
    abi.device_status()


@pytest.mark.parametrize("terms", [1, 2, 3])
@pytest.mark.parametrize("shape", [(17, 132), (640, 2560), (6912, 2560), (640, 9220), (2560, 8192)])
def test_row_alone_equals_row_among_others(ops, abi, shape, terms):
    """A row's result is the same to the bit whatever rows come with it, wherever it starts in memory and whether its scale
    is one number or one per output."""
    import torch
    out, inn = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(out + inn + terms)
    tiles = ops.int8_to_tiles(torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8))
    buf = torch.randn(5 * inn + 1, generator=g, device="cuda")
    x = buf[1:].view(5, inn)                                   # (off a 16-byte boundary)
    want = ops.bitlinear_forward(tiles, out, inn, x, terms, 0.037)
    vec = torch.full((out,), 0.037, device="cuda")
    for n in (1, 2, 3, 4):
        rows = x[:n].clone()
        assert torch.equal(ops.bitlinear_forward(tiles, out, inn, rows, terms, 0.037), want[:n]), n
        assert torch.equal(ops.bitlinear_forward(tiles, out, inn, rows, terms, wscale_vec=vec), want[:n]), n
        assert torch.equal(ops.bitlinear_forward(tiles, out, inn, x[:n], terms, 0.037), want[:n]), n
    abi.device_status()


@pytest.mark.parametrize("out,inn,rows,terms", [(12001, 8192, 5, 3), (3001, 1923, 13, 3), (640, 9000, 9, 1), (33001, 2048, 5, 1), (6912, 2560, 16, 1),
                                                (512, 8192, 8, 1), (1001, 4000, 7, 4), (600, 3000, 40, 1)])
def test_layer_call_equals_its_three_parts(ops, abi, out, inn, rows, terms):
    """Sums cleared by the quantiser or by a memset, products of one and of several launches, early and late starts: the call
    against quantiser, product and dequantiser called one by one, to the bit, twice over the same workspace."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(out + inn + rows)
    tiles = ops.int8_to_tiles(torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8))
    ws = torch.full((abi.lib.rotor_b200_bitlinear_workspace_bytes(out, inn, rows, terms),), 0x5A, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        x = torch.randn((rows, inn), generator=g, device="cuda")
        got = ops.bitlinear_forward(tiles, out, inn, x, terms, 0.037, workspace=ws)
        xq, sx, xsum = ops.quantize_rows(x, terms)
        acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, abi.VARIANT_AUTO)
        want = torch.empty_like(got)
        abi.check(abi.lib.rotor_b200_bitlinear_dequant(abi.ptr(acc), abi.ptr(sx), rows, terms, out, 0.037, None, abi.ptr(want), abi.stream()))
        assert torch.equal(got, want)
    abi.device_status()


@pytest.mark.parametrize("out,inn", [(3001, 1924), (600, 9216), (18432, 2560)])
@pytest.mark.parametrize("cols", [8, 9, 16, 17, 24, 25, 31, 32, 40, 41])
def test_products_of_a_few_dozen_columns(ops, abi, out, inn, cols):
    """One row tile a CTA, several, and the tensor-core tiles, on either side of every column count where the rule changes:
    the integers against a float64 product, in which they are exact; then the layer call, whose product may finish the rows,
    against its three parts to the bit, with one scale and one per output, rows off a 16-byte boundary, a row of zeros and rows
    with an infinity and a NaN."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(out + cols)
    w = torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8)
    tiles = ops.int8_to_tiles(w)
    q = torch.zeros((cols, abi.lib.rotor_b200_in_padded(inn)), dtype=torch.int8, device="cuda")
    q[:, :inn] = torch.randint(-128, 128, (cols, inn), generator=g, device="cuda", dtype=torch.int8)
    acc = ops.bitlinear_acc(tiles, out, inn, q, q.sum(1, dtype=torch.int32), abi.VARIANT_AUTO)
    assert torch.equal(acc.double(), q[:, :inn].double() @ w.double().T)
    x = torch.randn(cols * inn + 1, generator=g, device="cuda")[1:].view(cols, inn)
    x[1], x[2, 5], x[3, inn - 1] = 0.0, float("inf"), float("nan")
    vec = torch.rand(out, generator=g, device="cuda")
    for terms in (1, 3):
        rows = x[:max(1, cols // terms)]
        xq, sx, xsum = ops.quantize_rows(rows.clone(), terms)
        parts = ops.bitlinear_acc(tiles, out, inn, xq, xsum, abi.VARIANT_DP4A)
        for scales in (None, vec):
            want = torch.empty((len(rows), out), device="cuda")
            abi.check(abi.lib.rotor_b200_bitlinear_dequant(abi.ptr(parts), abi.ptr(sx), len(rows), terms, out, 0.037,
                                                           None if scales is None else abi.ptr(scales), abi.ptr(want), abi.stream()))
            got = ops.bitlinear_forward(tiles, out, inn, rows, terms, 0.037, wscale_vec=scales)
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(7.0), want.nan_to_num(7.0)), (terms, scales is None)
    abi.device_status()


def test_tcgen05_extreme_values(ops, abi):
    """-128 x -1 and 127 x +1 over K = 6912 on the tcgen05 path: sums stay exact in int32."""
    out, inn, ncols = 256, 6912, 256
    w = np.ones((out, inn), dtype=np.int8)
    w[::2] = -1
    tiles = ops.int8_to_tiles(w)
    q = np.full((ncols, inn), -128, dtype=np.int8)
    q[1::2] = 127
    xq, xsum = ops.to_device(q), ops.to_device(q.astype(np.int32).sum(axis=1).astype(np.int32))
    acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, abi.VARIANT_AUTO).cpu().numpy()
    assert np.array_equal(acc, q.astype(np.int32) @ w.astype(np.int32).T)
    abi.device_status()


def test_extreme_values_do_not_overflow(ops, abi):
    """All weights +1 and all activations -128 over the longest row the models use."""
    out, inn = 16, 28672
    w = np.ones((out, inn), dtype=np.int8)
    tiles = ops.int8_to_tiles(w)
    q = np.full((2, inn), -128, dtype=np.int8)
    q[1] = 127
    xq, xsum = ops.to_device(q), ops.to_device(q.astype(np.int32).sum(axis=1).astype(np.int32))
    for v in (abi.VARIANT_DP4A, abi.VARIANT_MMA):
        acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, v).cpu().numpy()
        assert (acc[0] == -128 * inn).all() and (acc[1] == 127 * inn).all()


@pytest.mark.parametrize("variant", ["dp4a", "mma"])
def test_config1_matches_reference_fixture(ops, abi, golden_dir, variant):
    """Config 1 (2560 -> 6912).  The fixture is what the unmodified reference returned."""
    z = np.load(os.path.join(golden_dir, "bitlinear_2560x6912.npz"))
    w, scale, x1, x16 = G.bitlinear_case()
    tiles = ops.packed_to_tiles(O.pack_ternary_matrix(w), 6912, 2560)
    v = abi.VARIANT_DP4A if variant == "dp4a" else abi.VARIANT_MMA
    # reference semantics: three-term activations reproduce the float path
    y = ops.bitlinear_forward(tiles, 6912, 2560, x1, 3, scale, variant=v).cpu().numpy()
    assert rel_err(y, z["y1"]) < TOL
    y16 = ops.bitlinear_forward(tiles, 6912, 2560, x16, 3, scale, variant=v).cpu().numpy()
    assert rel_err(y16, z["y16"]) < TOL
    # published semantics: single-term int8; the oracle quantises identically, so the
    # integers match exactly and the float32 output to rounding
    y_int = ops.bitlinear_forward(tiles, 6912, 2560, x16, 1, scale, variant=v).cpu().numpy()
    want, acc, _, _ = O.bitlinear_int(x16, w, scale, 1)
    assert np.array_equal(y_int, want)


def test_small_ragged_layer(ops, golden_dir):
    z = np.load(os.path.join(golden_dir, "bitlinear_small.npz"))
    w, scale, x = G.small_linear_case()
    tiles = ops.packed_to_tiles(O.pack_ternary_matrix(w), 20, 72)
    y = ops.bitlinear_forward(tiles, 20, 72, x, 3, scale).cpu().numpy()
    assert rel_err(y, z["y"]) < TOL


def test_per_row_scale_vector_and_host_seam(ops, abi):
    """The plug-in call shape: scales as a per-output vector, host arrays in and out
    (src/rotor/gpu_ternary.py:138-202)."""
    import ctypes
    rng = np.random.default_rng(8)
    w = O.synth_ternary(rng, 96, 384)
    tiles = ops.int8_to_tiles(w)
    x = rng.standard_normal(384).astype(np.float32)
    scales = rng.random(96).astype(np.float32) + 0.5
    y = np.zeros(96, dtype=np.float32)
    f32 = ctypes.POINTER(ctypes.c_float)
    st = abi.lib.rotor_b200_ternary_matmul_host(tiles.data_ptr(), scales.ctypes.data_as(f32),
                                                x.ctypes.data_as(f32), 384, 96, 3, y.ctypes.data_as(f32))
    assert st == 0
    want = O.backend_matvec(O.backend_codes(w), scales, x, 384, 96)
    assert rel_err(y, want) < TOL


def test_linearity_at_full_size(ops, abi):
    """Size-independent property at the XL shape (8192 -> 28672): acc(q1 + q2) = acc(q1) + acc(q2)."""
    out, inn = 28672, 8192
    rng = np.random.default_rng(77)
    w = O.synth_ternary(rng, out, inn)
    tiles = ops.int8_to_tiles(w)
    q = rng.integers(-60, 61, size=(2, inn), dtype=np.int8)
    q3 = np.concatenate([q, (q[0] + q[1])[None, :]], axis=0).astype(np.int8)
    xq, xsum = ops.to_device(q3), ops.to_device(q3.astype(np.int32).sum(axis=1).astype(np.int32))
    for v in (abi.VARIANT_DP4A, abi.VARIANT_MMA):
        acc = ops.bitlinear_acc(tiles, out, inn, xq, xsum, v).cpu().numpy()
        assert np.array_equal(acc[0] + acc[1], acc[2])
    # and a sampled exact check of 64 rows
    rows = rng.integers(0, out, size=64)
    want = q3.astype(np.int32) @ w[rows].astype(np.int32).T
    assert np.array_equal(acc[:, rows], want)


def test_errors_are_reported_not_swallowed(ops, abi):
    with pytest.raises(ValueError):
        ops.packed_to_tiles(np.zeros((4, 4), np.uint8), 16, 128)
    assert abi.lib.rotor_b200_bitlinear_acc(None, 16, 128, None, None, 1, None, 0, None) == 1
    import torch
    x = torch.zeros((1, 128), device="cuda")
    tiles = ops.int8_to_tiles(np.zeros((16, 128), np.int8))
    small = torch.empty(256, dtype=torch.uint8, device="cuda")
    y = torch.empty((1, 16), device="cuda")
    st = abi.lib.rotor_b200_bitlinear_forward(tiles.data_ptr(), 16, 128, x.data_ptr(), 1, 1, 1.0, None,
                                              y.data_ptr(), small.data_ptr(), 8, 0, None)
    assert st == 4   # workspace too small


def test_mma_sync_gemm_kept_as_comparison_path():
    """The mma.sync tiled GEMM (the pre-tcgen05 path) stays selectable with ROTOR_B200_NO_TCGEN05=1 and
    stays bit-exact.  The switch is read once per process, hence the child process."""
    import subprocess
    import sys
    code = r'''
import sys, numpy as np
sys.path[:0] = [%r, %r]
from oracle import bitlinear_np as O
from rotor_b200 import abi, ops
rng = np.random.default_rng(4)
for out, inn, ncols in ((640, 2560, 300), (6912, 384, 64)):
    w = O.synth_ternary(rng, out, inn)
    kpad = abi.lib.rotor_b200_in_padded(inn)
    q = np.zeros((ncols, kpad), dtype=np.int8)
    q[:, :inn] = rng.integers(-128, 128, size=(ncols, inn), dtype=np.int8)
    acc = ops.bitlinear_acc(ops.int8_to_tiles(w), out, inn, ops.to_device(q),
                            ops.to_device(q.astype(np.int32).sum(axis=1).astype(np.int32)), abi.VARIANT_AUTO).cpu().numpy()
    assert np.array_equal(acc, q[:, :inn].astype(np.int32) @ w.astype(np.int32).T)
print("ok")
''' % (os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
       os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rotor-rag_b200"))
    env = dict(os.environ, ROTOR_B200_NO_TCGEN05="1")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr[-2000:]


@pytest.mark.parametrize("shape", [(2560, 2560, 48), (2560, 2560, 49), (3001, 1923, 33), (8192, 9216, 33), (18432, 8192, 100), (8192, 9216, 128),
                                   (8192, 9216, 129), (38000, 1700, 127), (38000, 1700, 128), (600, 1536, 64), (600, 1408, 64)])
def test_products_of_up_to_128_columns_bit_exact(ops, abi, shape):
    """Both ways of adding the sums of a split product, and the 128-token variant split and whole, on either side of the
    column counts and K steps where they are chosen: the integers against a float64 product, in which they are exact."""
    import torch
    out, inn, ncols = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    w = torch.randint(-1, 2, (out, inn), generator=g, device="cuda", dtype=torch.int8)
    kpad = abi.lib.rotor_b200_in_padded(inn)
    q = torch.zeros((ncols, kpad), dtype=torch.int8, device="cuda")
    q[:, :inn] = torch.randint(-128, 128, (ncols, inn), generator=g, device="cuda", dtype=torch.int8)
    acc = ops.bitlinear_acc(ops.int8_to_tiles(w), out, inn, q, q.sum(1, dtype=torch.int32), abi.VARIANT_AUTO)
    assert torch.equal(acc, (q[:, :inn].double() @ w.double().T).to(torch.int32))
    abi.device_status()
