"""The matvec over up to sixteen vectors per pass (qmv_rows.cu) at the edges of its tiles, passes and splits, against the
dequantised weights in 64 bits (yule-core/src/dequant.rs:902-1009)."""

import numpy as np
import pytest

from test_gpu_runner import PREFILL_CFG
from yule_b200 import CudaTransformerRunner, DType, synth

pytestmark = pytest.mark.gpu

FORMATS = [DType.Q4_K, DType.Q5_K, DType.Q6_K, DType.Q8_0, DType.Q4_0]
# 22 bits of each x, fp32 sums, and random blocks whose minimum terms cancel most of the quants' (a factor of up to about
# four): sixteen units of 2^-22
BOUND = 16 * 2.0 ** -22


def multiply(backend, dtype, w, x, n_rows, x_stride, out_stride):
    batch, n_cols = x.shape
    xs = np.zeros((batch, x_stride), np.float32)
    xs[:, :n_cols] = x
    wh, xh = backend.upload(w), backend.upload(xs.reshape(-1))
    backend.prepare_weights(wh, dtype, n_rows, n_cols)
    oh = backend.upload(np.full(batch * out_stride, 7.0, np.float32))
    backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch, x_stride, out_stride)
    y = backend.download(oh, batch * out_stride).reshape(batch, out_stride)
    for h in (wh, xh, oh):
        backend.free(h)
    assert np.all(y[:, n_rows:] == 7.0)
    return y[:, :n_rows]


@pytest.mark.parametrize("dtype", FORMATS)
@pytest.mark.parametrize("n_rows,n_cols,batch", [
    (1, 256, 5),          # one row, one block
    (31, 512, 8),         # below a tile; two vector quads
    (33, 768, 9),         # past a tile; three blocks over a cluster; a third quad with one vector
    (1000, 2304, 12),     # nine blocks: clusters with unequal shares
    (65, 5120, 2),        # few vectors, long rows
    (96, 14336, 16),      # four quads, rows whose image does not fit: built in parts
    (300, 11008, 11),     # 43 blocks
])
def test_edges(backend, oracle, dtype, n_rows, n_cols, batch):
    w = synth.random_blocks(dtype, 900 + n_rows, n_rows * (n_cols // dtype.block_size))
    x = synth.normal(901 + batch, batch * n_cols).reshape(batch, n_cols)
    x *= np.float32(10.0) ** (np.arange(batch, dtype=np.float32)[:, None] % 7 - 3)
    x[0, : n_cols // 2] = 0.0  # blocks of zeros
    deq = oracle.dequant(int(dtype), w).reshape(n_rows, n_cols).astype(np.float64)
    ref = x.astype(np.float64) @ deq.T
    y = multiply(backend, dtype, w, x, n_rows, n_cols + 64, n_rows + 5)
    size = np.linalg.norm(ref, axis=1) if n_rows > 1 else (np.abs(x).astype(np.float64) @ np.abs(deq).T)[:, 0]
    assert np.all(np.linalg.norm(y - ref, axis=1) <= BOUND * size)
    # a vector with an infinity spoils nobody else's results
    bad = x.copy()
    bad[1, 3] = np.inf
    z = multiply(backend, dtype, w, bad, n_rows, n_cols + 64, n_rows + 5)
    others = np.arange(batch) != 1
    assert np.array_equal(z[others], y[others]) and not np.isfinite(z[1]).any()


@pytest.mark.parametrize("dtype", FORMATS)
@pytest.mark.parametrize("batch", [17, 40])
def test_more_vectors_than_a_pass(backend, oracle, dtype, batch):
    n_rows, n_cols = 200, 1024
    w = synth.random_blocks(dtype, 950, n_rows * (n_cols // dtype.block_size))
    x = synth.normal(951, batch * n_cols).reshape(batch, n_cols)
    ref = x.astype(np.float64) @ oracle.dequant(int(dtype), w).reshape(n_rows, n_cols).astype(np.float64).T
    y = multiply(backend, dtype, w, x, n_rows, n_cols, n_rows)
    assert np.all(np.linalg.norm(y - ref, axis=1) <= BOUND * np.linalg.norm(ref, axis=1))


@pytest.mark.parametrize("fmt,down", [(DType.Q4_K, DType.Q6_K), (DType.Q5_K, DType.Q5_K), (DType.Q6_K, DType.Q8_0), (DType.Q4_0, DType.Q4_0)])
@pytest.mark.parametrize("batch", [2, 6, 14, 20])
def test_decode_step_of_several_sequences(backend, fmt, down, batch):
    """Norm, Q/K/V, rotation and append, gate / up pair and residuals folded together, against one sequence at a time."""
    weights = synth.synthetic_model(PREFILL_CFG, seed=97, std=0.05, linear=fmt, ffn_down=down, output=down)
    toks = synth.tokens(98, batch * 4, PREFILL_CFG.vocab_size).reshape(batch, 4)
    run = CudaTransformerRunner(backend, PREFILL_CFG, weights, fused=1)
    single = CudaTransformerRunner(backend, PREFILL_CFG, weights, fused=1)
    got = [run.decode_batch(toks[:, i]) for i in range(4)]
    for b in {0, batch // 2, batch - 1}:
        single.reset()
        for i in range(4):
            want = single.decode_step(int(toks[b, i]))
            # each of the handful of matrices between the embedding and the logits is off by up to BOUND / 4 on either side
            assert np.linalg.norm(got[i][b] - want) <= 2 * BOUND * np.linalg.norm(want)
    single.close()
    run.close()
