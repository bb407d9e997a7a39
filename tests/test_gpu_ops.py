"""GPU parity of the op-level C ABI (quantizer, repack, dequant, quantized matmul) against the CPU checker."""
import ctypes as C

import numpy as np
import pytest

import oracle
from ruai_b200 import nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert nn.Device.is_available(), "these tests need a CUDA device"
    return nn.Device.cuda(0)


def same(cpu, got, tol):
    """tests/devices.rs:31-40."""
    cpu, got = np.asarray(cpu, np.float64), np.asarray(got, np.float64)
    assert cpu.shape == got.shape
    bad = ~((np.abs(cpu - got) <= tol * (1 + np.abs(cpu))) | (cpu == got))
    assert not bad.any(), f"{bad.sum()} of {bad.size} differ; worst {np.abs(cpu - got).max()}"


def bf16_round(a):
    """f32 -> bf16 (round to nearest even) as raw uint16, and the widened value."""
    b = np.ascontiguousarray(a, np.float32).view(np.uint32)
    r = ((b + 0x7FFF + ((b >> 16) & 1)) >> 16).astype(np.uint16)
    return r, (r.astype(np.uint32) << 16).view(np.float32)


def bf16_widen(r):
    return (np.asarray(r, np.uint16).astype(np.uint32) << 16).view(np.float32)


# ---- quantizer: bit exact with the checker (and so with layers.rs:112-165) ------------

@pytest.mark.parametrize("k,n", [(48, 17), (576, 192), (768, 2304), (4096, 1024)])
def test_quantize_int8_bit_exact(dev, k, n):
    w = oracle.synth_normal(7, k * 131 + n, (k, n))
    if n > 3:
        w[:, 3] = 0.0
    q, s = nn.quantize_int8_device(dev, w)
    qo, so = oracle.quantize_int8(w)
    assert np.array_equal(s, so) and np.array_equal(q, qo)


@pytest.mark.parametrize("k,n,g", [(8, 3, 4), (64, 20, 32), (576, 1536, 32), (4096, 512, 32), (64, 48, 16)])
def test_quantize_int4_bit_exact(dev, k, n, g):
    w = oracle.synth_normal(8, k * 131 + n, (k, n))
    w[:g, 0] = 0.0
    q, s = nn.quantize_int4_device(dev, w, g)
    qo, so = oracle.quantize_int4(w, g)
    assert np.array_equal(s, so) and np.array_equal(q, qo)


def test_quantizer_golden(dev, golden):
    q, s = nn.quantize_int8_device(dev, golden["q8_w"])
    assert np.array_equal(q, golden["q8_q"]) and np.array_equal(s, golden["q8_scale"])
    for tag in ("qa", "qb"):
        q, s = nn.quantize_int4_device(dev, golden[f"{tag}_w"], int(golden[f"{tag}_g"]))
        assert np.array_equal(q, golden[f"{tag}_packed"]) and np.array_equal(s, golden[f"{tag}_scale"])


def test_int4_group_must_divide_the_input_width(dev):
    """tests/quant.rs:136-140 through the C ABI."""
    with pytest.raises(ValueError, match="must be even and divide"):
        nn.quantize_int4_device(dev, np.zeros((30, 4), np.float32), 16)
    q = np.zeros((15, 4), np.int8)
    with pytest.raises(nn.RuaiError, match="must be even and divide"):
        nn.QWeight.int4(dev, q, np.zeros((2, 4), np.float32), 16)


# ---- repack round trip: bit exact -------------------------------------------------------

@pytest.mark.parametrize("k,n", [(64, 300), (33, 70), (32, 48), (576, 576), (4096, 1024), (1, 1)])
def test_repack_int8_round_trip(dev, k, n):
    rng = np.random.default_rng(k * 7 + n)
    q = rng.integers(-128, 128, (k, n), dtype=np.int8)
    s = rng.random(n, dtype=np.float32)
    w = nn.QWeight.int8(dev, q, s)
    q2, s2 = w.unpack()
    assert np.array_equal(q, q2) and np.array_equal(s, s2)


@pytest.mark.parametrize("k,n,g", [(64, 300, 32), (32, 70, 8), (64, 48, 16), (576, 1536, 32), (4096, 256, 32), (2, 1, 2)])
def test_repack_int4_round_trip_and_dequant(dev, k, n, g):
    rng = np.random.default_rng(k * 7 + n)
    q = rng.integers(-128, 128, (k // 2, n), dtype=np.int8)
    s = rng.random((k // g, n), dtype=np.float32)
    w = nn.QWeight.int4(dev, q, s, g)
    q2, s2 = w.unpack()
    assert np.array_equal(q, q2) and np.array_equal(s, s2)
    assert np.array_equal(w.dequant(), oracle.dequant_int4(q, s, g))  # tol 0, tests/devices.rs:491


# ---- quantized matmul: the reference's own GPU-vs-CPU cases (tests/devices.rs:444-502) ----

def run_matmul(dev, x, w, dtype, bias=None):
    if dtype == "f32":
        xt, xf = nn.Tensor.from_numpy(dev, x.astype(np.float32)), x.astype(np.float32)
    elif dtype == "f16":
        xh = x.astype(np.float16)
        xt, xf = nn.Tensor.from_numpy(dev, xh), xh.astype(np.float32)
    else:
        raw, xf = bf16_round(x)
        xt = nn.Tensor.from_numpy(dev, raw, rdtype=nn.BF16)
    bt = None if bias is None else nn.Tensor.from_numpy(dev, bias)
    y = nn._matmul_q(xt, w, bt).numpy()
    if dtype == "bf16":
        y = bf16_widen(y)
    return xf, y.astype(np.float32)


TOL = {"f32": 1e-4, "f16": 6e-3, "bf16": 3e-2}  # devices.rs: 1e-4, half_tol * 3


def round_to(y, dtype):
    if dtype == "f16":
        return y.astype(np.float16).astype(np.float32)
    if dtype == "bf16":
        return bf16_round(y)[1]
    return y


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("idx", [0, 1, 2])
def test_int8_matmul_reference_cases(dev, golden, idx, dtype):
    q, s = golden[f"i8_{idx}_q"], golden[f"i8_{idx}_s"]
    xf, y = run_matmul(dev, golden[f"i8_{idx}_x"], nn.QWeight.int8(dev, q, s), dtype)
    same(round_to(oracle.matmul_int8(xf, q, s), dtype), y, TOL[dtype])
    if dtype == "f32":
        same(golden[f"i8_{idx}_y"], y, 1e-4)


@pytest.mark.parametrize("dtype", ["f32", "f16", "bf16"])
@pytest.mark.parametrize("idx", [0, 1, 2])
def test_int4_matmul_reference_cases(dev, golden, idx, dtype):
    q, s, g = golden[f"i4_{idx}_q"], golden[f"i4_{idx}_s"], int(golden[f"i4_{idx}_g"])
    xf, y = run_matmul(dev, golden[f"i4_{idx}_x"], nn.QWeight.int4(dev, q, s, g), dtype)
    same(round_to(oracle.matmul_int4(xf, q, s), dtype), y, TOL[dtype])
    if dtype == "f32":
        same(golden[f"i4_{idx}_y"], y, 1e-4)


def test_int4_identity_reads_the_weights_back(dev, golden):
    """tests/quant.rs:55-57 on the device."""
    for tag in ("qa", "qb"):
        w, g = golden[f"{tag}_w"], int(golden[f"{tag}_g"])
        lin = nn.Linear(dev, w)
        lin.quantize_int4(g)
        assert sorted(lin.state_dict()) == ["weight_int4", "weight_int4_scale"]
        assert lin.dims() == w.shape
        got = lin.forward(nn.Tensor.from_numpy(dev, np.eye(w.shape[0], dtype=np.float32))).numpy()
        assert np.abs(got - golden[f"{tag}_want"]).max() < 1e-6


# ---- the microbenchmark grid: M in {1,4,16,64,512}, K=N in {576,1536,4096}, + [1,2048]@[2048,2048] ----

GRID = [(m, kn, kn) for kn in (576, 1536, 4096) for m in (1, 4, 16, 64)] + [(512, 576, 576), (512, 1536, 1536), (1, 2048, 2048),
        (3, 4096, 14336 // 4), (2, 14336 // 4, 4096), (16, 768, 2304), (7, 1000, 130)]


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", GRID)
def test_matmul_grid_f32(dev, m, k, n, bits):
    if bits == 4 and k % 32:
        k = (k // 32) * 32
    x = oracle.synth_normal(11, 0x30000000 + m * 31 + k, (m, k), 1.0)
    x[:, ::7] = 0.0  # the CPU path skips zero activations (cpu.rs:909, 1052)
    w = oracle.synth_normal(11, k * 65537 + n, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, want = nn.QWeight.int8(dev, q, s), oracle.matmul_int8(x, q, s)
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, want = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4(x, q, s)
    bias = oracle.synth_normal(11, 99, (n,))
    _, y = run_matmul(dev, x, qw, "f32", bias)
    same(want + bias, y, 1e-4)
    q2, s2 = qw.unpack()
    assert np.array_equal(q2, q) and np.array_equal(s2, s)


# the Llama-3-8B widths (hidden 4096, q/k/v 6144, MLP 14336) at prefill-sized row counts, ragged and full tiles
WIDE = [(17, 4096, 14336), (64, 4096, 6144), (128, 14336, 4096), (512, 4096, 4096), (17, 4096, 28672), (64, 4096, 28672), (512, 14336, 4096)]


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", WIDE)
def test_matmul_grid_8b_widths(dev, m, k, n, bits):
    x = oracle.synth_normal(13, 0x31000000 + m, (m, k), 1.0)
    w = oracle.synth_normal(13, k * 65537 + n, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, want = nn.QWeight.int8(dev, q, s), oracle.matmul_int8(x, q, s)
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, want = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4(x, q, s)
    _, y = run_matmul(dev, x, qw, "f32")
    # Quantized-Linear outputs: max-abs 1e-2 and 1e-3 relative to the output's scale, all but a sliver inside the 1e-4 * (1 + |y|)
    # of tests/devices.rs: what two bf16 pieces of the activations need.  The GEMM's pieces hold 22 bits and stay well inside;
    # test_gemm_every_tile has their bound.
    err = np.abs(want.astype(np.float64) - y).max()
    assert err <= 1e-2 and err <= 1e-3 * np.abs(want).max(), (err, np.abs(want).max())
    loose = ~(np.abs(want - y) <= 1e-4 * (1 + np.abs(want)))
    assert loose.mean() <= 1e-4, f"{loose.sum()} of {loose.size} outputs beyond the tests/devices.rs tolerance"


# 5..16 rows: the 16-row tile (weights streamed once).  Shapes chosen so that k splits over 1, 2, 4 and 8 CTAs, the last
# stage and the last column tile are ragged, and k is not a multiple of the group.
ROWS16 = [(9, 64, 48), (12, 96, 130), (16, 4096, 512), (13, 4096, 6144), (16, 14336, 4096), (10, 4096, 28672), (16, 1000, 130), (11, 1536, 1536),
          (5, 4096, 4096), (8, 14336, 4096), (6, 96, 70), (4, 14336, 4096),
          # 4M weights and more (what the 16-row kernel takes) with ragged edges: a last column tile of 76 / 4 / 2 columns, an
          # odd number of groups, a last stage of one group, k that is no multiple of 32 (int8), 8 splits of a long k
          (16, 4128, 1100), (9, 4000, 1100), (12, 8192, 516), (7, 2080, 2052), (16, 4096, 1026), (13, 1000, 4400)]


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", ROWS16)
def test_matmul_five_to_sixteen_rows(dev, m, k, n, bits):
    if bits == 4 and k % 32:
        k = (k // 32) * 32
    x = oracle.synth_normal(17, 0x32000000 + m * 31 + k, (m, k), 1.0)
    x[:, ::5] = 0.0
    w = oracle.synth_normal(17, k * 65537 + n, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, want = nn.QWeight.int8(dev, q, s), oracle.matmul_int8(x, q, s)
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, want = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4(x, q, s)
    bias = oracle.synth_normal(17, 98, (n,))
    _, y = run_matmul(dev, x, qw, "f32", bias)
    want = want + bias
    # the activations ride as two bf16 pieces (16 significant bits): the stated tolerance of quantized-Linear outputs,
    # and all but a sliver inside the 1e-4 of tests/devices.rs
    err = np.abs(want.astype(np.float64) - y).max()
    assert err <= 1e-2 and err <= 1e-3 * np.abs(want).max(), (err, np.abs(want).max())
    loose = ~(np.abs(want - y) <= 1e-4 * (1 + np.abs(want)))
    assert loose.mean() <= 1e-4, f"{loose.sum()} of {loose.size} outputs beyond the tests/devices.rs tolerance"
    for dtype in ("f16", "bf16"):
        xf, yh = run_matmul(dev, x, qw, dtype, bias)
        ref = oracle.matmul_int8(xf, q, s) if bits == 8 else oracle.matmul_int4(xf, q, s)
        same(round_to(ref + bias, dtype), yh, TOL[dtype])


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m", [1, 2, 3, 9])  # (one row has no splits)
def test_fixed_split_counts_give_the_same_product(dev, bits, m):
    """ruai_ctx_force_splits: the product does not depend on how many CTAs share k beyond the order of a few f32 additions
    (more splits than stages of k leave some CTAs of the cluster without work)."""
    k, n = 2048, 2304
    x = oracle.synth_normal(19, m, (m, k), 1.0)
    w = oracle.synth_normal(19, 2, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, want = nn.QWeight.int8(dev, q, s), oracle.matmul_int8(x, q, s)
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, want = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4(x, q, s)
    try:
        for splits in (0, 1, 2, 4, 8):
            dev.force_splits(splits)
            _, y = run_matmul(dev, x, qw, "f32")
            same(want, y, 1e-4 if m < 5 else 3e-4)
        with pytest.raises(Exception):
            dev.force_splits(9)
    finally:
        dev.force_splits(0)


@pytest.mark.slow
@pytest.mark.parametrize("m", [17, 64])
def test_matmul_head_width_int8(dev, m):
    """The 8B head [4096 -> 128256], int8 as the reference keeps it, at more than 16 rows (the GEMM path)."""
    k, n = 4096, 128256
    x = oracle.synth_normal(15, m, (m, k), 1.0)
    q, s = oracle.quantize_int8(oracle.synth_normal(15, 3, (k, n)))
    want = oracle.matmul_int8(x, q, s)
    _, y = run_matmul(dev, x, nn.QWeight.int8(dev, q, s), "f32")
    err = np.abs(want.astype(np.float64) - y).max()
    assert err <= 1e-2 and err <= 1e-3 * np.abs(want).max(), (err, np.abs(want).max())


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m", [1, 2, 5, 16, 40])
def test_matmul_non_finite_activations_propagate(dev, bits, m):
    """A NaN or an infinity in a row of x makes that row of the product non-finite, as f32 arithmetic on the CPU does
    (cpu.rs:1002-1029, 1035-1067); the other rows are unaffected."""
    k, n = 4096, 1024
    x = oracle.synth_normal(14, m, (m, k), 1.0)
    w = oracle.synth_normal(14, 2, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, f = nn.QWeight.int8(dev, q, s), oracle.matmul_int8
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, f = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4
    want = f(x, q, s)
    for bad in (np.nan, np.inf, -np.inf):
        xb = x.copy()
        xb[0, 1234] = bad
        _, y = run_matmul(dev, xb, qw, "f32")
        assert not np.isfinite(y[0]).any(), bad
        if m > 1:  # (5 to 16 rows: activations as two bf16 pieces, see test_matmul_five_to_sixteen_rows)
            same(want[1:], y[1:], 1e-4 if m < 5 else 3e-4)


@pytest.mark.parametrize("bits", [8, 4])
def test_matmul_bf16_activations(dev, bits):
    m, k, n = 16, 1536, 1536
    x = oracle.synth_normal(12, 1, (m, k), 1.0)
    w = oracle.synth_normal(12, 2, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        qw, f = nn.QWeight.int8(dev, q, s), oracle.matmul_int8
    else:
        q, s = oracle.quantize_int4(w, 32)
        qw, f = nn.QWeight.int4(dev, q, s, 32), oracle.matmul_int4
    xf, y = run_matmul(dev, x, qw, "bf16")
    same(bf16_round(f(xf, q, s))[1], y, 3e-2)


def test_linearity_and_determinism(dev):
    """Size-independent properties at a full-size shape: y(a*x1 + x2) = a*y(x1) + y(x2); repeat calls are bit identical."""
    k, n = 4096, 14336
    w = oracle.synth_normal(13, 5, (k, n))
    lin = nn.Linear(dev, w)
    lin.quantize_int4(32)
    x1 = oracle.synth_normal(13, 6, (1, k), 1.0)
    x2 = oracle.synth_normal(13, 7, (1, k), 1.0)
    y1 = lin.forward(nn.Tensor.from_numpy(dev, x1)).numpy()
    y2 = lin.forward(nn.Tensor.from_numpy(dev, x2)).numpy()
    y3 = lin.forward(nn.Tensor.from_numpy(dev, 2.0 * x1 + x2)).numpy()
    assert np.abs(y3 - (2.0 * y1 + y2)).max() < 1e-3 * np.abs(y3).max()
    again = lin.forward(nn.Tensor.from_numpy(dev, x1)).numpy()
    assert np.array_equal(again, y1)
    q, s = lin.int4
    same(oracle.matmul_int4(x1, q, s), y1, 1e-4)


# ---- training-side ops on the packed weights: input gradient and LoRA forward (layers.rs:169-190, ops.rs:705-734) ----

def _qw(dev, bits, k, n, seed, group=32):
    w = oracle.synth_normal(seed, k * 65537 + n, (k, n))
    if bits == 8:
        q, s = oracle.quantize_int8(w)
        return q, s, nn.QWeight.int8(dev, q, s)
    q, s = oracle.quantize_int4(w, group)
    return q, s, nn.QWeight.int4(dev, q, s, group)


@pytest.mark.parametrize("bits,group", [(8, 32), (4, 32), (4, 16)])
@pytest.mark.parametrize("m,k,n", [(1, 64, 48), (3, 576, 1536), (5, 4096, 1024), (2, 96, 130)])
def test_grad_input_matches_checker_and_is_the_adjoint(dev, m, k, n, bits, group):
    q, s, qw = _qw(dev, bits, k, n, 21, group)
    g = oracle.synth_normal(21, 7, (m, n), 1.0)
    want = oracle.matmul_q_grad_input(bits, g, q, s, group)
    got = nn.matmul_q_grad_input(nn.Tensor.from_numpy(dev, g), qw).numpy()
    same(want, got, 1e-4)
    # adjoint identity with the forward op of this library: <g, x @ W> == <g @ W^T, x>
    x = oracle.synth_normal(21, 8, (m, k), 1.0)
    y = nn._matmul_q(nn.Tensor.from_numpy(dev, x), qw).numpy().astype(np.float64)
    lhs, rhs = float((g * y).sum()), float((got.astype(np.float64) * x).sum())
    assert abs(lhs - rhs) <= 2e-4 * max(abs(lhs), np.abs(g).sum() * 1e-3)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n,rank", [(1, 64, 48, 4), (4, 576, 1536, 8), (2, 4096, 1024, 16), (3, 96, 130, 3)])
def test_lora_forward_matches_checker(dev, m, k, n, rank, bits):
    q, s, qw = _qw(dev, bits, k, n, 22)
    x = oracle.synth_normal(22, 1, (m, k), 1.0)
    a = oracle.synth_normal(22, 2, (k, rank), 1.0 / np.sqrt(k))
    b = oracle.synth_normal(22, 3, (rank, n), 0.05)
    bias = oracle.synth_normal(22, 4, (n,))
    scale = 16.0 / rank
    T = lambda v: nn.Tensor.from_numpy(dev, v)
    for bb in (None, bias):
        want = oracle.linear_lora_forward(bits, x, q, s, a, b, scale, bb)
        got = nn.linear_lora_forward(T(x), qw, T(a), T(b), scale, None if bb is None else T(bb)).numpy()
        same(want, got, 1e-4)
    # B = 0 (a fresh adapter, layers.rs:93): the output is the base layer's
    zero = np.zeros((rank, n), np.float32)
    got = nn.linear_lora_forward(T(x), qw, T(a), T(zero), scale).numpy()
    assert np.array_equal(got, nn._matmul_q(T(x), qw).numpy())


# ---- few rows on the dot-product units: edges of the tiles of columns, of the warps' ranges of k, of the blocks of one exponent ----

@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("k,n,rows", [(32, 4, (1, 2, 8)), (64, 8, (1, 3, 16)), (96, 36, (1, 4, 9)), (544, 132, (1, 2, 3, 4, 8, 13, 16)), (1056, 1300, (1, 2, 5, 16)),
                                      (1536, 1664, (2, 4, 8, 16)), (2080, 2500, (1,)), (4128, 4900, (1,)), (4096, 4736, (1,)), (14336, 96, (1,)), (512, 28672, (1,))])
def test_few_rows_against_float64(dev, k, n, rows, bits, dtype):
    """x is rounded to half of 2^-22 (int8: 2^-27) of the largest magnitude of its block of 32 (128) at the most, the sums are f32: errors
    below that, summed over the block's weights, and 2^-20 of the sum of the products' magnitudes."""
    if bits == 8:  # a ragged last chunk, rows of x that are not aligned, an odd number of columns
        k -= 5
        n -= 1
    q, s, qw = _qw(dev, bits, k, n, 51)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    bias = oracle.synth_normal(51, 1, (n,))
    for m in rows:
        x = oracle.synth_normal(51, m, (m, k), 1.0) * np.exp2(np.arange(k) // 32 % 23 - 11).astype(np.float32)  # blocks of very different size
        xf, got = run_matmul(dev, x, qw, dtype, bias)
        want, mag = xf.astype(np.float64) @ wd + bias, np.abs(xf).astype(np.float64) @ np.abs(wd) + np.abs(bias)
        # int8: a block of one exponent is 128 consecutive k of a warp's range: no larger than twice 128 neighbours
        lo, hi = (0, 32) if bits == 4 else (224, 256)
        top = np.stack([np.abs(xf[:, max(0, i - lo):i + hi]).max(1) for i in range(0, k, 32)], 1)
        rounding = np.repeat(top, 32, 1)[:, :k].astype(np.float64) @ np.abs(wd) * 2.0 ** (-22 if bits == 4 else -27)
        bound = rounding + 2.0 ** -20 * mag + (2.0 ** -8 * np.abs(want) if dtype == "bf16" else 0.0) + 1e-30
        assert (np.abs(got - want) <= bound).all(), (m, (np.abs(got - want) / bound).max())


@pytest.mark.parametrize("k", [32769, 40000])
def test_long_rows_of_int8_stay_f32(dev, k):
    """Beyond k = 32768 the activations are multiplied as they are: small ones beside a large one whose weights are zero are not lost."""
    n = 64
    rng = np.random.default_rng(k)
    q = rng.integers(1, 128, (k, n)).astype(np.int8)
    q[::128] = 0
    s = np.full(n, 0.01, np.float32)
    x = np.ones((1, k), np.float32)
    x[0, ::128] = 2.0 ** 30
    _, got = run_matmul(dev, x, nn.QWeight.int8(dev, q, s), "f32", None)
    want = x.astype(np.float64) @ (q.astype(np.float64) * s)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("k,n,rows", [(2080, 1100, (2, 3, 4, 8, 9, 16)), (1568, 132, (2, 4, 9, 16)), (4000, 900, (2, 3, 8, 16)), (1024, 19460, (1,))])
def test_narrow_tensor_core_kernels_against_float64(dev, k, n, rows, bits):
    """Just past the line where the dot-product kernel ends, below the 4M weights of the 16-row one (and one row of int8 that stays with the tensor
    cores): ragged columns and k, every number of splits.  x is rounded to half of 2^-20 of the largest of its 32 (int4), 2^-27 of the largest
    of its row (int8), and f32 sums leave 2^-20 of the products' magnitudes."""
    if bits == 8:
        k -= 5
        n -= 1
    q, s, qw = _qw(dev, bits, k, n, 53)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    bias = oracle.synth_normal(53, 1, (n,))
    try:
        for m in rows:
            x = oracle.synth_normal(53, m, (m, k), 1.0) * np.exp2(np.arange(k) // 32 % 15 - 7).astype(np.float32)
            want, mag = x.astype(np.float64) @ wd + bias, np.abs(x).astype(np.float64) @ np.abs(wd) + np.abs(bias)
            if bits == 4:
                top = np.abs(x).reshape(m, k // 32, 32).max(2)
                rounding = np.repeat(top, 32, 1).astype(np.float64) @ np.abs(wd) * 2.0 ** -20
            else:
                rounding = np.abs(x).max(1, keepdims=True) * np.abs(wd).sum(0) * 2.0 ** -27
            for splits in (0, 1, 2, 4, 8):
                dev.force_splits(splits)
                _, got = run_matmul(dev, x, qw, "f32", bias)
                bound = rounding + 2.0 ** -20 * mag
                assert (np.abs(got - want) <= bound).all(), (m, splits, (np.abs(got - want) / bound).max())
    finally:
        dev.force_splits(0)


# ---- the GEMM's tiles: edges of rows, columns and k, every split of k ----

@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", [(17, 64, 128), (64, 96, 132), (65, 4160, 300), (128, 2016, 256), (129, 544, 516), (300, 1504, 1500), (513, 224, 2564)])
def test_gemm_tiles_against_float64(dev, m, k, n, bits):
    """Both fp16 pieces of x carry 22 bits, sums are f32: errors below 2^-20 of the sum of the products' magnitudes."""
    if bits == 8:
        k -= 7  # a ragged last chunk
    q, s, qw = _qw(dev, bits, k, n, 31)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    x = oracle.synth_normal(31, m, (m, k), 1.0) * np.exp2(np.arange(m) % 40 - 20).astype(np.float32)[:, None]  # rows of very different size
    want, mag = x.astype(np.float64) @ wd, np.abs(x).astype(np.float64) @ np.abs(wd)
    xt = nn.Tensor.from_numpy(dev, x)
    try:
        for splits in (0, 1, 2, 3, 5, 7, 8):
            dev.force_splits(splits)
            got = nn._matmul_q(xt, qw).numpy().astype(np.float64)
            assert (np.abs(got - want) <= 2.0 ** -20 * mag + 1e-30).all(), (splits, (np.abs(got - want) / mag).max())
    finally:
        dev.force_splits(0)


@pytest.mark.parametrize("dtype,bits,ratio,quantum", [("f32", 4, 28, 2.0 ** -50), ("f32", 8, 20, 2.0 ** -38), ("bf16", 4, 100, 0.0), ("bf16", 8, 28, 0.0), ("f16", 4, 14, 0.0), ("f16", 8, 14, 0.0)])
@pytest.mark.parametrize("m,k,n", [(37, 544, 300), (150, 1504, 516)])
def test_gemm_small_elements_beside_large_ones(dev, m, k, n, dtype, bits, ratio, quantum):
    """Every row has elements 2^ratio times the others whose weights are zero: what the others keep is seen alone.  A scaled row's pieces
    round to half their quantum of the row's largest; 16-bit elements are exact, and the output is rounded to their type."""
    w = oracle.synth_normal(35, k * 65537 + n, (k, n))
    w[5::97] = 0.0
    q, s = oracle.quantize_int8(w) if bits == 8 else oracle.quantize_int4(w, 32)
    qw = nn.QWeight.int8(dev, q, s) if bits == 8 else nn.QWeight.int4(dev, q, s, 32)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    x = oracle.synth_normal(35, m, (m, k), 1.0)
    x = np.where(np.abs(x) < 0.5, 0.5, x).astype(np.float32)  # none further below the row's largest than stated
    x[:, 5::97] = 2.0 ** ratio
    xf, got = run_matmul(dev, x, qw, dtype)
    want, mag = xf.astype(np.float64) @ wd, np.abs(xf).astype(np.float64) @ np.abs(wd)
    bound = 2.0 ** -20 * mag + 0.5 * quantum * np.abs(xf).max(1, keepdims=True).astype(np.float64) * np.abs(wd).sum(0)
    bound += {"f32": 0.0, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype] * np.abs(want) + 1e-7
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


TILES = [(256, 128), (128, 128), (128, 64)]


def _against_float64(dev, dtype, bits, m, k, n, seed):
    """Sums in f32 of products that hold 22 bits of x: errors below 2^-20 of the sum of the products' magnitudes, and the rounding of a
    16-bit output."""
    if bits == 8:
        k -= 7  # a ragged last chunk
    q, s, qw = _qw(dev, bits, k, n, seed)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    x, bias = oracle.synth_normal(seed, m, (m, k), 1.0), oracle.synth_normal(seed, 1, (n,))
    xf, got = run_matmul(dev, x, qw, dtype, bias)
    want, mag = xf.astype(np.float64) @ wd + bias, np.abs(xf).astype(np.float64) @ np.abs(wd) + np.abs(bias)
    bound = 2.0 ** -20 * mag + {"f32": 0.0, "f16": 2.0 ** -11, "bf16": 2.0 ** -8}[dtype] * np.abs(want) + 1e-7
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / bound).max()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("m,k,n", [(17, 64, 128), (64, 96, 132), (129, 544, 516), (300, 1504, 1500), (513, 224, 2564),
                                   # several tiles per CTA, of three, one and four stages: the rings and barriers go on from tile to tile
                                   (2053, 160, 4900), (1700, 64, 6404), (2053, 256, 4900)])
def test_gemm_every_tile(dev, tile, m, k, n, bits):
    try:
        dev.force_tile(*tile)
        _against_float64(dev, "f32", bits, m, k, n, 41)
        with pytest.raises(nn.RuaiError, match="tile"):
            dev.force_tile(256, 64)
    finally:
        dev.force_tile(0, 0)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("m,k,n", [(17, 96, 132), (37, 1504, 1500), (129, 544, 516), (513, 224, 2564), (2053, 160, 4900)])
def test_gemm_half_precision_activations(dev, tile, m, k, n, dtype, bits):
    try:
        dev.force_tile(*tile)
        _against_float64(dev, dtype, bits, m, k, n, 42)
    finally:
        dev.force_tile(0, 0)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", [(2000, 576, 3072), (2000, 576, 960), (4000, 1120, 1536), (3000, 4096, 2560)])
def test_gemm_again_and_again(dev, m, k, n, bits):
    """Several tiles per CTA, of an odd number of stages among others: every run gives the same bits, and the status stays clean."""
    q, s, qw = _qw(dev, bits, k, n, 45)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    x = oracle.synth_normal(45, m, (m, k), 1.0)
    xt = nn.Tensor.from_numpy(dev, x)
    first = nn._matmul_q(xt, qw).numpy()
    want, mag = x.astype(np.float64) @ wd, np.abs(x).astype(np.float64) @ np.abs(wd)
    assert (np.abs(first - want) <= 2.0 ** -20 * mag + 1e-30).all()
    for _ in range(12):
        ys = [nn._matmul_q(xt, qw) for _ in range(8)]
        dev.synchronize()
        assert all(np.array_equal(y.numpy(), first) for y in ys[::3])


@pytest.mark.parametrize("m,n", [(88320, 384), (88320, 300)])
def test_gemm_of_one_group_over_many_tiles(dev, m, n):
    """k of one scale group and a dozen column blocks per CTA: the scales' ring goes round with one group per stage."""
    q, s, qw = _qw(dev, 4, 32, n, 34)
    x = oracle.synth_normal(34, 1, (m, 32), 1.0)
    got = nn._matmul_q(nn.Tensor.from_numpy(dev, x), qw).numpy()
    rows = np.r_[0:m:37, m - 1]
    wd = qw.dequant().astype(np.float64)
    want, mag = x[rows].astype(np.float64) @ wd, np.abs(x[rows]).astype(np.float64) @ np.abs(wd)
    assert (np.abs(got[rows] - want) <= 2.0 ** -20 * mag + 1e-30).all()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", [(7, 32, 16), (18, 64, 40), (19, 96, 17), (63, 96, 17), (65, 160, 300), (200, 2048, 1000)])
def test_grad_input_tiles_against_float64(dev, m, k, n, bits):
    """f32 sums of n terms, each rounded three times: errors below (n + 3) 2^-24 of the sum of the magnitudes."""
    if bits == 8:
        k -= 5
    q, s, qw = _qw(dev, bits, k, n, 32)
    wd = q.astype(np.float64) * s if bits == 8 else qw.dequant().astype(np.float64)
    g = oracle.synth_normal(32, m, (m, n), 1.0)
    want, mag = g.astype(np.float64) @ wd.T, np.abs(g).astype(np.float64) @ np.abs(wd).T
    got = nn.matmul_q_grad_input(nn.Tensor.from_numpy(dev, g), qw).numpy().astype(np.float64)
    assert (np.abs(got - want) <= (n + 3) * 2.0 ** -24 * mag + 1e-30).all()


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", [(19, 512, 512), (256, 2048, 2048), (64, 2048, 4096), (512, 4096, 1500), (40, 1024, 600)])
def test_grad_input_error_does_not_grow_with_the_columns(dev, m, k, n, bits):
    """Sums of 16 terms whose additions' rests are carried on: sixteen roundings of a growing sum, sqrt(16 / 2) 2^-24 / sqrt(3) = 0.97e-7 of
    the result in the 2-norm at the most (each rounding uniform within half a unit in the last place)."""
    q, s, qw = _qw(dev, bits, k, n, 36)
    wd = (q * s).astype(np.float64) if bits == 8 else qw.dequant().astype(np.float64)
    g = oracle.synth_normal(36, m, (m, n), 1.0)
    want = g.astype(np.float64) @ wd.T
    got = nn.matmul_q_grad_input(nn.Tensor.from_numpy(dev, g), qw).numpy().astype(np.float64)
    assert np.linalg.norm(got - want) <= 1.0e-7 * np.linalg.norm(want)


@pytest.mark.parametrize("bits", [8, 4])
@pytest.mark.parametrize("m,k,n", [(19, 64, 2000), (65, 4096, 300), (600, 4096, 80)])
def test_grad_input_infinities_and_nans(dev, m, k, n, bits):
    """A row with an infinity sums to infinities, one with a NaN or with both infinities to NaN; the other rows are what they were."""
    q, s, qw = _qw(dev, bits, k, n, 37)
    g = oracle.synth_normal(37, m, (m, n), 1.0)
    T = lambda v: nn.matmul_q_grad_input(nn.Tensor.from_numpy(dev, v), qw).numpy()
    plain = T(g)
    bad = g.copy()
    bad[0, 3], bad[1, n - 1], bad[2, 7], bad[m - 1, 5], bad[m - 1, n - 5] = np.inf, -np.inf, np.nan, np.inf, -np.inf
    bad[3, 0] = bad[3, 1] = 3e38  # overflows, or not, by the weights' signs
    got = T(bad)
    wd = (q * s).astype(np.float64) if bits == 8 else qw.dequant().astype(np.float64)
    with np.errstate(invalid="ignore", over="ignore"):
        want = bad[[0, 1, 2, m - 1]].astype(np.float64) @ wd.T
    for row, w in zip(got[[0, 1, 2, m - 1]], want):
        assert np.array_equal(np.isnan(row), np.isnan(w)) and np.array_equal(row[np.isinf(w)], w[np.isinf(w)].astype(np.float32))
    others = np.r_[4:m - 1]
    assert np.allclose(got[others], plain[others], rtol=1e-5, atol=1e-6)


class Capturing:
    """A context on a stream of its own, whose work can be captured into a graph."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        self.stream, self.graph, self.exec = C.c_void_p(), C.c_void_p(), C.c_void_p()
        assert self.cu.cuStreamCreate(C.byref(self.stream), 1) == 0  # not ordered with the legacy stream
        self.dev = nn.Device.__new__(nn.Device)
        self.dev.ordinal, self.dev.L, self.dev.ctx = 0, nn._lib.load(), C.c_void_p()
        nn._lib.check(self.dev.L.ruai_ctx_create(0, self.stream, C.byref(self.dev.ctx)))

    def begin(self):
        assert self.cu.cuStreamBeginCapture_v2(self.stream, 1) == 0  # of this thread

    def end(self):
        return self.cu.cuStreamEndCapture(self.stream, C.byref(self.graph))

    def replay(self):
        if not self.exec:
            assert self.cu.cuGraphInstantiateWithFlags(C.byref(self.exec), self.graph, C.c_ulonglong(0)) == 0
        assert self.cu.cuGraphLaunch(self.exec, self.stream) == 0
        self.dev.synchronize()

    def close(self):
        if self.exec:
            self.cu.cuGraphExecDestroy(self.exec)
        if self.graph:
            self.cu.cuGraphDestroy(self.graph)
        nn._lib.check(self.dev.L.ruai_ctx_destroy(self.dev.ctx))
        assert self.cu.cuStreamDestroy_v2(self.stream) == 0


@pytest.fixture()
def capturing(dev):
    c = Capturing()
    yield c
    c.close()


@pytest.mark.parametrize("m,k,n", [(256, 4096, 1024), (300, 1800, 1024), (20, 64, 300)])
def test_grad_input_in_a_graph(dev, capturing, m, k, n):
    """The gradient can be captured on a fresh context, and its graph replayed after the context's scratch has moved."""
    d = capturing.dev
    q, s, qw = _qw(d, 8, k, n, 38)
    wd = (q * s).astype(np.float64)
    gs = [oracle.synth_normal(38, i, (m, n), 1.0) for i in (1, 2)]
    g, dx = nn.Tensor.from_numpy(d, gs[0]), nn.Tensor(d, (m, k), np.float32, nn.F32)
    capturing.begin()
    rc = d.L.ruai_matmul_q_grad_input(d.ctx, g.ptr, qw.h, dx.ptr, m)
    assert capturing.end() == 0 and rc == 0

    def check(v):
        want = v.astype(np.float64) @ wd.T
        assert np.linalg.norm(dx.numpy() - want) <= 1.0e-7 * np.linalg.norm(want)

    capturing.replay()
    check(gs[0])
    _, _, big = _qw(d, 8, 4096, 256, 39)
    nn._matmul_q(nn.Tensor.from_numpy(d, np.full((1000, 4096), 3.0, np.float32)), big)  # its scratch is larger than a context's first
    d.check(d.L.ruai_memcpy_h2d(d.ctx, g.ptr, np.ascontiguousarray(gs[1]).ctypes.data_as(C.c_void_p), g.nbytes))
    capturing.replay()
    check(gs[1])
    for t in (g, dx, qw, big):
        t.free()


def test_results_while_their_memory_goes_round(dev):
    """Results dropped while they are queued, on one stream: their blocks come back several times."""
    q, s, qw = _qw(dev, 8, 2048, 2048, 33)
    xs = [nn.Tensor.from_numpy(dev, oracle.synth_normal(33, i, (256, 2048), 1.0)) for i in range(3)]
    want = [nn._matmul_q(x, qw).numpy() for x in xs]
    for r in range(120):
        i = r % 3
        for j in range(3):
            nn._matmul_q(xs[j], qw)
        assert np.array_equal(nn._matmul_q(xs[i], qw).numpy(), want[i])


def test_freed_tensors_are_reused_only_after_a_wait(dev):
    """A tensor freed through its own context while another context's stream has yet to read it: its block comes back to the first one only
    after that read."""
    other = nn.Device(0)
    m, k, n = 2048, 4096, 4096
    _, _, qw = _qw(other, 8, k, n, 43)
    data = oracle.synth_normal(43, 1, (m, k), 1.0)
    xs = [nn.Tensor.from_numpy(dev, data) for _ in range(3)]  # 32 MB each
    out, busy = (nn.Tensor(other, (m, n), np.float32, nn.F32) for _ in range(2))

    def product(x, y):
        other.check(other.L.ruai_matmul_q(other.ctx, nn.F32, x.ptr, qw.h, None, y.ptr, m))

    product(xs[0], out)
    want = out.numpy()
    other.check(other.L.ruai_memcpy_h2d(other.ctx, out.ptr, np.zeros_like(want).ctypes.data_as(C.c_void_p), out.nbytes))
    for _ in range(150):  # about 20 ms
        product(xs[0], busy)
    product(xs[1], out)
    freed = {t.ptr.value for t in xs[1:]}
    for t in xs[1:]:
        t.free()
    again = [nn.Tensor(dev, (m, k), np.float32, nn.F32) for _ in range(2)]
    for t in again:
        dev.check(dev.L.ruai_memcpy_h2d(dev.ctx, t.ptr, np.full_like(data, np.nan).ctypes.data_as(C.c_void_p), t.nbytes))
    got = out.numpy()
    assert {t.ptr.value for t in again} == freed  # they did come back
    assert np.array_equal(got, want)
    for t in (out, busy, qw):
        t.free()
    nn._lib.check(other.L.ruai_ctx_destroy(other.ctx))


def test_memory_freed_in_a_capture_or_twice_is_refused(dev, capturing):
    d = capturing.dev
    p, q = C.c_void_p(), C.c_void_p()
    d.check(d.L.ruai_malloc(d.ctx, 4096, C.byref(p)))
    capturing.begin()
    assert d.L.ruai_free(d.ctx, p) == nn._lib.ERR_CUDA
    assert capturing.end() != 0 and not capturing.graph  # as a wait for the capturing stream ends it
    d.check(d.L.ruai_free(d.ctx, p))
    assert d.L.ruai_free(d.ctx, p) == nn._lib.ERR_CUDA and dev.L.ruai_free(dev.ctx, p) == nn._lib.ERR_CUDA
    d.check(d.L.ruai_malloc(d.ctx, 4096, C.byref(q)))
    d.check(d.L.ruai_free(d.ctx, q))
    y = nn._matmul_q(nn.Tensor.from_numpy(dev, np.ones((3, 64), np.float32)), _qw(dev, 8, 64, 48, 44)[2])  # no error is left over for the next launch
    assert np.isfinite(y.numpy()).all()
