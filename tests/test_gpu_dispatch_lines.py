"""Lines of the dispatch, from both sides: dependent one-vector matvecs over many rows on half-size CTAs (qmv_digits.cu), activation rows that
share a CTA in the GEMM's re-layout (qgemm_tc.cu)."""

import numpy as np
import pytest

from conftest import guarded_rel_err, REL_TOL
from test_gpu_runner import make_oracle_model
from yule_b200 import CudaB200Backend, CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [DType.Q4_K, DType.Q8_0, DType.Q4_0, DType.Q6_K])
@pytest.mark.parametrize("vocab", [29984, 30000, 30016])
def test_output_matrix_in_the_token_step(backend, oracle, dtype, vocab):
    cfg = ModelConfig(dim=512, n_layers=1, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=vocab, ff_dim=512, max_seq_len=16)
    weights = synth.synthetic_model(cfg, seed=7, std=0.05, linear=DType.Q8_0, output=dtype)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    got, want = run.prefill([3, 17, 4]), ref.prefill([3, 17, 4])
    for t in (29983, 5):
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()  # 22-bit activations, fp32 sums over 512 columns: some 1e-6
        got, want = run.decode_step(t), ref.decode_step(t)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    run.close()


@pytest.mark.parametrize("dtype", [DType.Q4_K, DType.Q4_0])
@pytest.mark.parametrize("dim,ff,vocab", [(2048, 15104, 512), (2304, 15104, 512), (4096, 512, 30016), (4352, 512, 30016)])
def test_columns_of_a_pair_and_of_an_output_matrix(backend, oracle, dtype, dim, ff, vocab):
    """30208 rows of gate and up, 30016 of an output matrix: half-size CTAs up to 2048 and 4096 columns."""
    cfg = ModelConfig(dim=dim, n_layers=1, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=vocab, ff_dim=ff, max_seq_len=16)
    weights = synth.synthetic_model(cfg, seed=8, std=0.05, linear=dtype)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    got, want = run.prefill([3, 17]), ref.prefill([3, 17])
    for t in (500, 5):
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
        got, want = run.decode_step(t), ref.decode_step(t)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    run.close()


@pytest.mark.parametrize("dtype", [DType.Q4_K, DType.Q8_0])
@pytest.mark.parametrize("cols", [256, 4096, 4352, 8192, 8448, 16384, 16640])
@pytest.mark.parametrize("batch,pad", [(255, 0), (257, 0), (300, 4), (384, 8)])
def test_re_layout(backend, oracle, dtype, cols, batch, pad):
    """Two rows per CTA from 296 padded rows on; rows that are not packed; a padded last tile."""
    rows, stride = 40, cols + pad
    w, x = synth.random_quantized(dtype, 11, rows * cols), synth.normal(12, batch * stride)
    wh, xh, oh = backend.upload(w), backend.upload(x), backend.allocate(batch * rows * 4)
    backend.quantized_matmul_batched(wh, xh, oh, rows, cols, dtype, batch, stride, rows)
    y = backend.download(oh, batch * rows).reshape(batch, rows)
    for b in (0, 1, 2, batch // 2, batch - 2, batch - 1):
        ref = oracle.qmv(int(dtype), w, x[b * stride:b * stride + cols], rows, cols)
        assert guarded_rel_err(y[b], ref) <= REL_TOL
        assert np.abs(y[b] - ref).max() <= 1e-5 * np.abs(ref).max()
    for h in (wh, xh, oh):
        backend.free(h)


def test_long_prompt_through_two_row_re_layout(backend, oracle):
    cfg = ModelConfig(dim=512, n_layers=2, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=600, ff_dim=768, max_seq_len=400)
    weights = synth.synthetic_model(cfg, seed=9, std=0.05, linear=DType.Q4_K, ffn_down=DType.Q6_K)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    prompt = synth.tokens(10, 333, cfg.vocab_size)
    got, want = run.prefill(prompt), ref.prefill(list(prompt))
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    run.close()


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("rows,batch", [(4352, 9), (4608, 10), (4608, 12)])  # 119, 126 and 126 Mi weights
def test_nine_to_twelve_vectors_over_a_large_matrix(oracle, rows, batch, captured):
    """The matvec over all of them in one pass, which needs no scratch: also as the first call of a context, inside a capture."""
    cols = 28672
    b = CudaB200Backend(0)
    w, x = synth.random_quantized(DType.Q4_K, 21, rows * cols), synth.normal(22, batch * cols)
    wh, xh, oh = b.upload(w), b.upload(x), b.allocate(batch * rows * 4)
    if captured:
        b.graph_begin()
    b.quantized_matmul_batched(wh, xh, oh, rows, cols, DType.Q4_K, batch)
    if captured:
        b.graph_launch(b.graph_end())
    y = b.download(oh, batch * rows).reshape(batch, rows)
    b.close()
    for i in (0, batch - 1):
        assert guarded_rel_err(y[i], oracle.qmv(int(DType.Q4_K), w, x[i * cols:(i + 1) * cols], rows, cols)) <= REL_TOL


def test_nine_to_twelve_vectors_are_as_exact_as_eight(backend, oracle):
    """The same arithmetic up to twelve vectors, whatever the size of the matrix: exact quants with their middle taken out, sums in fp32.  Against 64 bits
    that is 0.8e-7 to 1.2e-7; the truncating accumulators of the GEMM give 2.2e-7 to 2.8e-7.  1.3: two draws of the same rounding errors over 128 rows of
    eight or more vectors differ by a few percent (a 2-norm of 1000 or more independent errors)."""
    rows, cols = 4608, 28672  # 126 Mi weights
    w, x = synth.random_quantized(DType.Q4_K, 31, rows * cols), synth.normal(32, 12 * cols)
    wh, xh, oh = backend.upload(w), backend.upload(x), backend.allocate(12 * rows * 4)
    some = np.r_[0:64, rows - 64:rows]
    row_bytes = w.size // rows
    dense = np.stack([oracle.dequant(int(DType.Q4_K), w[r * row_bytes:(r + 1) * row_bytes]) for r in some]).astype(np.float64)
    exact = x.reshape(12, cols).astype(np.float64) @ dense.T
    error = {}
    for batch in (8, 9, 12):
        backend.quantized_matmul_batched(wh, xh, oh, rows, cols, DType.Q4_K, batch)
        y = backend.download(oh, batch * rows).reshape(batch, rows)[:, some]
        error[batch] = np.linalg.norm(y - exact[:batch]) / np.linalg.norm(exact[:batch])
    for h in (wh, xh, oh):
        backend.free(h)
    assert error[9] <= 1.3 * error[8] and error[12] <= 1.3 * error[8], error
