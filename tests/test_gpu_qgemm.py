"""Tensor-core GEMM path of quantized_matmul_batched (eight or more activation rows) against the
scalar CPU restatement of Yule's per-row dot product (yule-gpu/src/cpu.rs:149-175), row by row."""

import numpy as np
import pytest

from yule_b200 import DType, synth

from conftest import REL_TOL, guarded_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def gemm_for_small_batches(monkeypatch):
    """By default the GEMM takes over from 16 (Q4_K) or 32 (other formats) activation rows; these tests
    want it from 8, its smallest tile."""
    monkeypatch.setenv("YULE_GEMM_MIN_BATCH", "8")


def run(backend, w, x, n_rows, n_cols, batch, x_stride=None, out_stride=None, dtype=DType.Q4_K):
    x_stride = x_stride or n_cols
    out_stride = out_stride or n_rows
    xs = np.zeros((batch, x_stride), np.float32)
    xs[:, :n_cols] = x.reshape(batch, n_cols)
    wh, xh = backend.upload(w), backend.upload(xs.reshape(-1))
    oh = backend.upload(np.full(batch * out_stride, 7.0, np.float32))
    backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch, x_stride, out_stride)
    backend.synchronize()
    y = backend.download(oh, batch * out_stride).reshape(batch, out_stride)
    for h in (wh, xh, oh):
        backend.free(h)
    return y


@pytest.mark.parametrize("n_rows,n_cols,batch", [
    (128, 256, 8),        # one tile, one super-block per row
    (256, 512, 32),       # a full 32-row activation tile
    (1000, 1024, 33),     # ragged rows and one activation row past a tile
    (513, 2048, 64),
    (300, 2048, 200),     # two 128-row activation tiles, the second padded
    (4096, 4096, 128),
    (2048, 5632, 16),     # the TinyLlama down-projection shape
])
def test_gemm_matches_scalar_reference(backend, oracle, n_rows, n_cols, batch):
    w = synth.random_blocks(DType.Q4_K, 300 + n_rows, n_rows * (n_cols // 256))
    x = synth.normal(301 + batch, batch * n_cols)
    y = run(backend, w, x, n_rows, n_cols, batch)
    worst = 0.0
    for b in range(0, batch, max(1, batch // 24)):  # up to ~24 activation rows, spread over the tiles
        ref = oracle.qmv(int(DType.Q4_K), w, x[b * n_cols:(b + 1) * n_cols], n_rows, n_cols)
        worst = max(worst, guarded_rel_err(y[b], ref))
    assert worst <= REL_TOL
    # Against an exact (float64) product of the dequantised weights the error stays near the fp32
    # accumulation floor: the fp16 hi/lo split keeps 22 bits, the tensor core truncates its fp32 sums.
    W = oracle.dequant(int(DType.Q4_K), w).astype(np.float64).reshape(n_rows, n_cols)
    X = x.astype(np.float64).reshape(batch, n_cols)
    scale = np.sqrt((X ** 2).sum(1))[:, None] * np.sqrt((W ** 2).sum(1))[None, :]
    assert (np.abs(y - X @ W.T) / scale).max() <= 4e-6


def test_gemm_strides_and_untouched_padding(backend, oracle):
    n_rows, n_cols, batch = 200, 512, 9
    w = synth.random_blocks(DType.Q4_K, 41, n_rows * (n_cols // 256))
    x = synth.normal(42, batch * n_cols)
    y = run(backend, w, x, n_rows, n_cols, batch, x_stride=n_cols + 64, out_stride=n_rows + 24)
    for b in range(batch):
        ref = oracle.qmv(int(DType.Q4_K), w, x[b * n_cols:(b + 1) * n_cols], n_rows, n_cols)
        assert guarded_rel_err(y[b, :n_rows], ref) <= REL_TOL
    assert np.all(y[:, n_rows:] == 7.0)  # the gap between output rows is not written


def test_gemm_rows_with_very_different_magnitudes(backend, oracle):
    """Every activation row gets its own power-of-two scale: tiny, huge and zero rows in one tile."""
    n_rows, n_cols, batch = 256, 1024, 12
    w = synth.random_quantized(DType.Q4_K, 43, n_rows * n_cols)
    x = synth.normal(44, batch * n_cols).reshape(batch, n_cols)
    x[1] *= 1e-6
    x[2] *= 1e5
    x[3] = 0.0
    x[4, 5] = 3e4  # one outlier far above the rest of its row
    y = run(backend, w, x.reshape(-1), n_rows, n_cols, batch)
    for b in range(batch):
        ref = oracle.qmv(int(DType.Q4_K), w, x[b], n_rows, n_cols)
        assert guarded_rel_err(y[b], ref) <= REL_TOL
    assert np.all(y[3] == 0.0)


def test_gemm_equals_matvec_path(backend):
    """Batch 8 (GEMM) and batch 4 + 4 (tensor-pipe matvec) agree to the parity tolerance."""
    n_rows, n_cols = 1024, 2048
    w = synth.random_quantized(DType.Q4_K, 45, n_rows * n_cols)
    x = synth.normal(46, 8 * n_cols)
    y8 = run(backend, w, x, n_rows, n_cols, 8)
    y4 = np.concatenate([run(backend, w, x[:4 * n_cols], n_rows, n_cols, 4),
                         run(backend, w, x[4 * n_cols:], n_rows, n_cols, 4)])
    assert guarded_rel_err(y8.reshape(-1), y4.reshape(-1)) <= REL_TOL


@pytest.mark.parametrize("dtype", [DType.Q6_K, DType.Q8_0, DType.Q4_0, DType.Q4_K, DType.Q5_K, DType.Q5_0, DType.Q4_1, DType.Q5_1,
                                   DType.Q8_1, DType.Q3_K, DType.Q2_K])
@pytest.mark.parametrize("n_rows,n_cols,batch", [(200, 512, 9), (513, 2048, 64), (1024, 1024, 200)])
def test_generic_format_gemm(backend, oracle, monkeypatch, dtype, n_rows, n_cols, batch):
    """Every format but Q4_K (and Q4_K when forced) goes through the kernel whose producers dequantise with the
    bit-exact per-element routine and split the weight into fp16 hi + lo."""
    monkeypatch.setenv("YULE_GEMM_GENERIC", "1")
    w = synth.random_blocks(dtype, 500 + n_rows, n_rows * (n_cols // dtype.block_size))
    x = synth.normal(501 + batch, batch * n_cols)
    y = run(backend, w, x, n_rows, n_cols, batch, dtype=dtype)
    W = oracle.dequant(int(dtype), w).astype(np.float64).reshape(n_rows, n_cols)
    X = x.astype(np.float64).reshape(batch, n_cols)
    scale = np.sqrt((X ** 2).sum(1))[:, None] * np.sqrt((W ** 2).sum(1))[None, :]
    assert (np.abs(y - X @ W.T) / scale).max() <= 4e-6
    for b in range(0, batch, max(1, batch // 8)):
        ref = oracle.qmv(int(dtype), w, x[b * n_cols:(b + 1) * n_cols], n_rows, n_cols)
        assert guarded_rel_err(y[b], ref) <= REL_TOL


@pytest.mark.parametrize("dtype", [DType.Q4_K, DType.Q8_0, DType.Q6_K])
@pytest.mark.parametrize("n_rows,n_cols,batch,forced", [
    (256, 4096, 32, None),    # two tiles, sixteen super-blocks: four parts of four
    (200, 2816, 16, None),    # eleven super-blocks: parts of six and five, ragged rows
    (1280, 8192, 32, None),   # the Q/K/V slice of a 70B-class layer on eight GPUs
    (2560, 2048, 24, 8),      # 160 work items: some CTAs take two
])
def test_column_split(backend, oracle, monkeypatch, dtype, n_rows, n_cols, batch, forced):
    """With few row tiles and long rows the columns of a tile are split over several CTAs; the warp that stores its
    part last adds the parts in their order.  Same result as the unsplit kernel to fp32 rounding, the same bits on
    every launch (the tickets return to zero), parity with the scalar reference."""
    w = synth.random_blocks(dtype, 700 + n_rows, n_rows * (n_cols // dtype.block_size))
    x = synth.normal(701 + batch, batch * n_cols)
    if forced:
        monkeypatch.setenv("YULE_GEMM_KSPLIT", str(forced))
    y = run(backend, w, x, n_rows, n_cols, batch, dtype=dtype)
    again = run(backend, w, x, n_rows, n_cols, batch, dtype=dtype)
    assert np.array_equal(y, again)
    monkeypatch.setenv("YULE_GEMM_KSPLIT", "1")
    whole = run(backend, w, x, n_rows, n_cols, batch, dtype=dtype)
    assert not np.array_equal(y, whole), "the split did not take place"
    assert np.abs(y - whole).max() <= 4e-6 * np.abs(whole).max()
    for b in (0, batch // 2, batch - 1):
        ref = oracle.qmv(int(dtype), w, x[b * n_cols:(b + 1) * n_cols], n_rows, n_cols)
        assert guarded_rel_err(y[b], ref) <= REL_TOL


@pytest.mark.parametrize("dtype", [DType.Q8_0, DType.Q4_0, DType.Q6_K, DType.Q5_K])
def test_extreme_block_scales(backend, oracle, dtype):
    """The unpacking of the generic kernel in half precision: scales from the smallest subnormal to just below 64, where d·2^10 is
    still a half (above it the product with a quant is outside the operands' range), and quants at both ends."""
    n_rows, n_cols, batch = 130, 512, 70
    size, per_row = dtype.size_of_block, n_cols // dtype.block_size
    w = np.array(synth.random_blocks(dtype, 31, n_rows * per_row)).reshape(-1, size).copy()
    at = 208 if dtype == DType.Q6_K else 0
    exps = np.arange(n_rows) % 28
    d = np.repeat((2.0 ** -24 * 2.0 ** exps * 1.37).astype(np.float16), per_row)  # 2^-24 … 2^3
    w[:, at:at + 2] = d.view(np.uint8).reshape(-1, 2)
    if dtype == DType.Q5_K:
        w[:, 2:4] = d.view(np.uint8).reshape(-1, 2)
    if dtype in (DType.Q6_K, DType.Q5_K):  # d times a scale times a quant stays below 64
        big = np.repeat(exps, per_row) > 15
        w[big, at:at + 2] = 0
        if dtype == DType.Q5_K:
            w[big, 2:4] = 0
    # a weight of 64 or more is outside the operands' range: 127 d, 8 d below it, or quants of 1
    if dtype == DType.Q8_0:
        w[np.repeat(exps, per_row) > 22, 2:] = 1
    if dtype == DType.Q4_0:
        w[np.repeat(exps, per_row) > 26, 2:] = 0x99
    w[0, at + 2 if at == 0 else 0] = 0xFF
    w[1, at + 2 if at == 0 else 0] = 0x80
    w = w.reshape(-1)
    x = synth.normal(32, batch * n_cols).reshape(batch, n_cols)
    deq = oracle.dequant(int(dtype), w).reshape(n_rows, n_cols).astype(np.float64)
    ref = x.astype(np.float64) @ deq.T
    wh, xh, oh = backend.upload(w), backend.upload(x.reshape(-1)), backend.allocate(batch * n_rows * 4)
    backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
    y = backend.download(oh, batch * n_rows).reshape(batch, n_rows)
    for h in (wh, xh, oh):
        backend.free(h)
    # row by row: 22 bits of x and of each weight (weights below 2^-24 in the lo term lose theirs: 2^-25 each, after the scaling
    # by 2^10), fp32 sums
    bound = 16 * 2.0 ** -22 * np.abs(x).astype(np.float64) @ np.abs(deq).T + 2.0 ** -35 * np.abs(x).sum(1)[:, None]
    assert np.all(np.abs(y - ref) <= bound)


@pytest.mark.parametrize("dtype,units", [(DType.Q8_0, 3), (DType.Q6_K, 3), (DType.Q4_K, 6)])
@pytest.mark.parametrize("batch", [40, 200])
def test_error_against_64_bits(backend, oracle, dtype, units, batch):
    """In units of 2^-24 of the result (2-norm).  Operands of 22 bits cost one unit, the fp32 sums of 32 stages of 64 columns one, the
    truncation of at most four additions of large products in the tensor core less than one; Q4_K sums q and its minimum apart,
    each twice as large as their difference.  (Measured 2.1 and 4.8; with the small products in turn with the large ones 5.4 and 7.7 at 200 rows.)"""
    n_rows, n_cols = 256, 2048
    w = synth.random_quantized(dtype, 95, n_rows * n_cols)
    x = synth.normal(96, batch * n_cols)
    y = run(backend, w, x, n_rows, n_cols, batch, dtype=dtype)
    if dtype == DType.Q6_K:  # d·sc·q in 64 bits (the oracle's values are rounded to 32)
        blocks = np.asarray(w).reshape(-1, 210)
        scale = blocks[:, 208:].copy().view(np.float16).astype(np.float64) * blocks[:, 192:208].copy().view(np.int8)
        scale = np.repeat(scale, 16, axis=1).reshape(n_rows, n_cols)
        exact = np.where(scale == 0, 0, np.rint(oracle.dequant(int(dtype), w).reshape(n_rows, n_cols) / np.where(scale == 0, 1, scale))) * scale
    else:
        exact = oracle.dequant(int(dtype), w).reshape(n_rows, n_cols).astype(np.float64)
    want = x.reshape(batch, n_cols).astype(np.float64) @ exact.T
    error = np.linalg.norm(y - want) / np.linalg.norm(want) * 2 ** 24
    assert error <= units, error
