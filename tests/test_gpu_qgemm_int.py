"""The GEMM of Q8_0, Q4_0, Q5_K and Q6_K whose W operand is an exact integer (csrc/qgemm_int.cu): against 64 bits and against the dequantising kernel that
takes these formats where this one cannot (csrc/qgemm_tc.cu)."""

import numpy as np
import pytest

from yule_b200 import CudaB200Backend, DType, synth

from conftest import guarded_rel_err, REL_TOL

pytestmark = pytest.mark.gpu

FORMATS = [DType.Q8_0, DType.Q4_0, DType.Q5_K, DType.Q6_K]


@pytest.fixture(autouse=True)
def gemm_for_small_batches(monkeypatch):
    monkeypatch.setenv("YULE_GEMM_MIN_BATCH", "8")


def run(backend, w, x, n_rows, n_cols, dtype, planar=True):
    batch = x.size // n_cols
    wh, xh, oh = backend.upload(w), backend.upload(x), backend.upload(np.full(batch * n_rows, 7.0, np.float32))
    if planar:
        backend.prepare_weights(wh, dtype, n_rows, n_cols)
    backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
    y = backend.download(oh, batch * n_rows).reshape(batch, n_rows)
    for h in (wh, xh, oh):
        backend.free(h)
    return y


def weights64(oracle, dtype, w, n_rows, n_cols):
    """The weights in 64 bits: block scales times whole numbers, nothing rounded."""
    b = np.asarray(w).reshape(-1, dtype.size_of_block)
    half = lambda at: b[:, at:at + 2].copy().view(np.float16).astype(np.float64)  # noqa: E731
    v = oracle.dequant(int(dtype), w).reshape(len(b), -1).astype(np.float64)
    if dtype == DType.Q6_K:
        s = np.repeat(half(208) * b[:, 192:208].copy().view(np.int8), 16, axis=1)
        v = np.where(s == 0, 0, np.rint(v / np.where(s == 0, 1, s))) * s
    elif dtype == DType.Q5_K:
        lo, hi = b[:, 4:8], b[:, 8:12]
        sc = np.concatenate([lo & 63, (b[:, 12:16] & 15) | (lo >> 6 << 4)], 1).astype(np.float64)
        mn = np.concatenate([hi & 63, (b[:, 12:16] >> 4) | (hi >> 6 << 4)], 1).astype(np.float64)
        bits = (b[:, 16:48, None] >> np.arange(8)) & 1                       # fifth bit of (column, sub-block)
        nib = b[:, 48:].reshape(-1, 4, 32)
        q = np.stack([nib & 15, nib >> 4], 2).reshape(-1, 8, 32) | (bits.transpose(0, 2, 1) << 4)
        v = ((half(0) * sc)[:, :, None] * q - (half(2) * mn)[:, :, None]).reshape(len(b), -1)
    return v.reshape(n_rows, n_cols)


@pytest.mark.parametrize("dtype", FORMATS)
@pytest.mark.parametrize("n_rows,n_cols,batch", [
    (1, 256, 8),          # one row, one super-block
    (129, 512, 32),       # one row past a tile, a full tile of 32 activation rows
    (200, 1280, 33),      # five super-blocks: the box ring wraps in the middle of a row
    (513, 2304, 64),
    (300, 2048, 200),     # two activation tiles of 128, the second padded; columns split over CTAs
    (20000, 512, 129),    # several tiles per CTA
    (256, 14336, 24),     # long rows, split columns
])
def test_against_64_bits_and_the_dequantising_kernel(backend, oracle, monkeypatch, dtype, n_rows, n_cols, batch):
    w = synth.random_blocks(dtype, 900 + n_rows, n_rows * (n_cols // dtype.block_size))
    x = synth.normal(901 + batch, batch * n_cols)
    y = run(backend, w, x, n_rows, n_cols, dtype)
    assert np.array_equal(y, run(backend, w, x, n_rows, n_cols, dtype))
    monkeypatch.setenv("YULE_GEMM_GENERIC", "1")
    other = run(backend, w, x, n_rows, n_cols, dtype)
    W = weights64(oracle, dtype, w, n_rows, n_cols)
    X = x.reshape(batch, n_cols).astype(np.float64)
    want = X @ W.T
    scale = np.sqrt((X ** 2).sum(1))[:, None] * np.sqrt((W ** 2).sum(1))[None, :]
    # operands of 22 bits, fp32 sums: a unit or two of 2^-22 of |x||w| each
    assert (np.abs(y - want) / scale).max() <= 1e-6
    assert (np.abs(y - other) / scale).max() <= 2e-6
    for b in (0, batch - 1):
        assert guarded_rel_err(y[b], oracle.qmv(int(dtype), w, x[b * n_cols:(b + 1) * n_cols], n_rows, n_cols)) <= REL_TOL


@pytest.mark.parametrize("dtype", FORMATS)
@pytest.mark.parametrize("batch", [20, 40, 200])
def test_no_less_precise_than_the_dequantising_kernel(backend, oracle, monkeypatch, dtype, batch):
    """2-norm against 64 bits on weights as a quantiser makes them; 1.1: two draws of the same rounding errors."""
    n_rows, n_cols = 256, 2048
    w = synth.random_quantized(dtype, 95, n_rows * n_cols)
    x = synth.normal(96, batch * n_cols)
    want = x.reshape(batch, n_cols).astype(np.float64) @ weights64(oracle, dtype, w, n_rows, n_cols).T
    error = lambda y: np.linalg.norm(y - want) / np.linalg.norm(want)  # noqa: E731
    now = error(run(backend, w, x, n_rows, n_cols, dtype))
    monkeypatch.setenv("YULE_GEMM_GENERIC", "1")
    assert now <= 1.1 * error(run(backend, w, x, n_rows, n_cols, dtype))


def test_scales_of_any_size(backend, oracle):
    """No range is lost: block scales from the smallest subnormal to the largest half, quants at both ends, and zero."""
    n_rows, n_cols, batch = 160, 512, 40
    for dtype in FORMATS:
        per_row = n_cols // dtype.block_size
        w = np.array(synth.random_blocks(dtype, 31, n_rows * per_row)).reshape(-1, dtype.size_of_block).copy()
        at = 208 if dtype == DType.Q6_K else 0
        d = 2.0 ** (-24 + np.arange(n_rows) % 39) * 1.37
        d[0] = 0
        d = np.repeat(d.astype(np.float16), per_row)
        w[:, at:at + 2] = d.view(np.uint8).reshape(-1, 2)
        if dtype == DType.Q5_K:
            w[:, 2:4] = np.roll(d, 3 * per_row).view(np.uint8).reshape(-1, 2)
        quants = {DType.Q8_0: 2, DType.Q4_0: 2, DType.Q5_K: 48, DType.Q6_K: 0}[dtype]
        w[per_row, quants:quants + 8] = 0xFF
        w[2 * per_row, quants:quants + 8] = 0x80
        w = w.reshape(-1)
        x = synth.normal(32, batch * n_cols)
        y = run(backend, w, x, n_rows, n_cols, dtype)
        W = weights64(oracle, dtype, w, n_rows, n_cols)
        X = x.reshape(batch, n_cols).astype(np.float64)
        # Q5_K: the centred quants and their offset may each be some 63·31·d + 63·dmin
        big = np.abs(W)
        if dtype == DType.Q5_K:
            big += (63 * 31 * np.repeat(d.astype(np.float64), 256) + 63 * np.repeat(np.roll(d, 3 * per_row).astype(np.float64), 256)).reshape(n_rows, n_cols)
        assert np.all(np.abs(y - X @ W.T) <= 16 * 2.0 ** -22 * (np.abs(X) @ big.T) + 1e-30), dtype


def test_rows_of_very_different_size(backend, oracle):
    """Every activation row has its own scale: tiny, huge and zero rows in one tile."""
    n_rows, n_cols, batch = 256, 1024, 12
    x = synth.normal(44, batch * n_cols).reshape(batch, n_cols)
    x[1] *= 1e-6
    x[2] *= 1e5
    x[3] = 0.0
    x[4, 5] = 3e4
    for dtype in FORMATS:
        w = synth.random_quantized(dtype, 43, n_rows * n_cols)
        y = run(backend, w, x.reshape(-1), n_rows, n_cols, dtype)
        for b in range(batch):
            assert guarded_rel_err(y[b], oracle.qmv(int(dtype), w, x[b], n_rows, n_cols)) <= REL_TOL
        assert np.all(y[3] == 0.0)


def test_q6_k_without_its_planar_copy(backend, oracle):
    """Stays on the kernel that reads the raw blocks."""
    n_rows, n_cols = 300, 768
    w = synth.random_blocks(DType.Q6_K, 5, n_rows * 3)
    x = synth.normal(6, 40 * n_cols)
    a, b = (run(backend, w, x, n_rows, n_cols, DType.Q6_K, planar=p) for p in (False, True))
    assert np.abs(a - b).max() <= 2e-6 * np.abs(a).max()


@pytest.mark.parametrize("dtype", FORMATS)
@pytest.mark.parametrize("batch", [17, 20, 24, 32, 33, 48])
def test_both_sides_of_the_line_to_the_matvec(oracle, monkeypatch, dtype, batch):
    """Where the call goes by itself, and as the first call of a context inside a capture, where the GEMM's scratch cannot be allocated and the matvec over
    sixteen vectors a pass, which needs none, keeps what it takes."""
    monkeypatch.delenv("YULE_GEMM_MIN_BATCH")
    for n_rows, n_cols in ((256, 512), (4224, 4096)):
        w, x = synth.random_quantized(dtype, 51, n_rows * n_cols), synth.normal(52, batch * n_cols)
        got = []
        for captured in (False, True):
            b = CudaB200Backend(0)
            wh, xh, oh = b.upload(w), b.upload(x), b.allocate(batch * n_rows * 4)
            b.prepare_weights(wh, dtype, n_rows, n_cols)
            takes = batch <= 32 or n_rows * n_cols > 17 << 20 or dtype in (DType.Q4_0, DType.Q5_K)
            if captured and takes:
                b.graph_begin()
                b.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
                b.graph_launch(b.graph_end())
            else:
                b.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
            got.append(b.download(oh, batch * n_rows).reshape(batch, n_rows))
            b.close()
        for i in (0, batch - 1):
            assert guarded_rel_err(got[0][i], oracle.qmv(int(dtype), w, x[i * n_cols:(i + 1) * n_cols], n_rows, n_cols)) <= REL_TOL
        assert np.abs(got[0] - got[1]).max() <= 2e-6 * np.abs(got[0]).max()
