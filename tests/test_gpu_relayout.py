"""Activations of few rows to the GEMM's operands by clusters of CTAs (gemm_xprep_cluster_kernel in csrc/qgemm_tc.cu)."""

import numpy as np
import pytest

from yule_b200 import CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cols,batch", [
    (768, 20),      # fewer blocks of 256 columns than CTAs in a cluster: one CTA per row
    (1024, 20),     # a block per CTA
    (1280, 17),     # shares of one and two blocks, padding rows
    (2304, 64),
    (4096, 100),    # 65 rows and more, laid out and no more: one CTA per row (the prompts below have the clusters of two)
    (4608, 250),
    (9472, 128),
    (9728, 128),
    (16384, 40),    # 32 warps of two rows
    (16640, 40),    # one row per CTA
    (32768, 32),    # 32 warps of one
    (33024, 32),    # too long
])
def test_every_share_of_a_row(backend, oracle, n_cols, batch):
    n_rows, dtype = 40, DType.Q8_0
    w = synth.random_blocks(dtype, 3, n_rows * n_cols // 32)
    x = synth.normal(4, batch * n_cols).reshape(batch, n_cols).copy()
    for b in range(batch):  # the largest of a row in each block in turn, and rows of very different size
        x[b, (b * 256 + 7 * b) % n_cols] = 300.0 * (-1) ** b
        x[b] *= 2.0 ** (b % 41 - 20)
    x[1], x[2, : n_cols // 2] = 0, 0
    wh, xh, oh = backend.upload(w), backend.upload(x), backend.allocate(batch * n_rows * 4)
    backend.prepare_weights(wh, dtype, n_rows, n_cols)
    backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
    y = backend.download(oh, batch * n_rows).reshape(batch, n_rows)
    for h in (wh, xh, oh):
        backend.free(h)
    q = np.asarray(w).reshape(-1, 34)
    W = (q[:, :2].copy().view(np.float16).astype(np.float64) * q[:, 2:].view(np.int8)).reshape(n_rows, n_cols)
    X = x.astype(np.float64)
    scale = np.sqrt((X ** 2).sum(1))[:, None] * np.sqrt((W ** 2).sum(1))[None, :]
    # operands of 22 bits, fp32 sums: a unit or two of 2^-22 of |x||w| each
    assert not y[1].any()
    assert (np.abs(y - X @ W.T) <= 1e-6 * scale).all()


@pytest.mark.parametrize("dim,ff,n", [(1280, 4608, 20), (1280, 4608, 60), (1280, 4608, 100), (1280, 4608, 250), (1024, 28672, 20), (8192, 1024, 30)])
def test_norm_and_swiglu(backend, dim, ff, n):
    """A prompt's logits against those of its tokens one after another, which no GEMM sees."""
    cfg = ModelConfig(dim=dim, n_layers=2, n_heads=4, n_kv_heads=4, head_dim=64, vocab_size=300, ff_dim=ff, max_seq_len=n + 8)
    weights = synth.synthetic_model(cfg, seed=21, std=0.03, linear=DType.Q4_K)
    prompt = synth.tokens(22, n, cfg.vocab_size)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    got = run.prefill(prompt)
    run.reset()
    for t in prompt:
        want = run.decode_step(t)
    run.close()
    # fp32 rounding (some 2^-22 of a layer's output) through two layers, of the largest logit
    assert np.abs(got - want).max() <= 2e-5 * np.abs(want).max()
