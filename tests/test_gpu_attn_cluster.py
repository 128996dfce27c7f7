"""Decode attention on thread-block clusters (csrc/attn_cluster.cu) at the sizes where its split changes: fewer positions than
CTAs, a tile of 32 and its neighbours, one cluster and several, the line to the kernel with splits, full contexts."""

import numpy as np
import pytest

from test_gpu_runner import make_oracle_model
from yule_b200 import CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu

# A score is a sum of head_dim products, off by at most head_dim * 2^-24 of the sum of their magnitudes (about sqrt(head_dim) after the
# scaling, for N(0, 1) values): 8e-5 at 128 in the worst case, a tenth of that with roundings of random sign; the weights carry it on.
TOL = 1e-5


def attention64(q, K, V, n_heads, n_kv, hd):
    q, K, V = (a.astype(np.float64) for a in (q.reshape(n_heads, hd), K, V))
    out = np.empty((n_heads, hd))
    for h in range(n_heads):
        kv = h // (n_heads // n_kv)
        s = K[:, kv * hd:(kv + 1) * hd] @ q[h] / np.sqrt(hd)
        e = np.exp(s - s.max())
        out[h] = e @ V[:, kv * hd:(kv + 1) * hd] / e.sum()
    return out.reshape(-1)


@pytest.mark.parametrize("hd,n_heads,n_kv,seqs", [
    (64, 32, 4, (1, 2, 7, 8, 9, 31, 33, 255, 256, 257, 1000, 5119, 5120, 5121)),
    (128, 32, 8, (1, 3, 32, 64, 65, 511, 513, 768, 769, 2560, 2561)),
    (128, 64, 8, (5, 100, 1023)), (64, 4, 4, (6, 300, 1500)), (128, 2, 1, (4, 700)), (64, 16, 8, (33, 600))])
def test_one_query(backend, hd, n_heads, n_kv, seqs):
    stride = n_kv * hd + 4  # rows that are not packed
    for seq in seqs:
        q, K, V = synth.normal(seq, n_heads * hd), synth.normal(seq + 1, seq * stride), synth.normal(seq + 2, seq * stride)
        q *= 3  # some positions dominate
        handles = [backend.upload(a) for a in (q, K, V)] + [backend.allocate(n_heads * hd * 4)]
        qh, kh, vh, oh = handles
        for _ in range(2):  # the second call finds the tickets of the first
            backend.multihead_attention(qh, kh, vh, oh, hd, seq, n_heads, n_kv, stride)
        y = backend.download(oh, n_heads * hd)
        ref = attention64(q, K.reshape(seq, stride), V.reshape(seq, stride), n_heads, n_kv, hd)
        assert np.abs(y - ref).max() <= TOL * np.abs(ref).max(), (hd, n_heads, n_kv, seq)
        for h in handles:
            backend.free(h)


@pytest.mark.parametrize("hd,n_heads,n_kv,ctx,prompt", [(64, 4, 2, 24, 3), (64, 8, 1, 40, 30), (64, 8, 4, 300, 250), (128, 4, 4, 130, 120),
                                                        (128, 8, 2, 800, 760), (64, 16, 2, 700, 500)])
def test_runner_up_to_the_full_context(backend, oracle, hd, n_heads, n_kv, ctx, prompt):
    cfg = ModelConfig(dim=256, n_layers=2, n_heads=n_heads, n_kv_heads=n_kv, head_dim=hd, vocab_size=512, ff_dim=512, max_seq_len=ctx)
    weights = synth.synthetic_model(cfg, seed=3, std=0.08, linear=DType.Q8_0)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    tokens = [(7 * i + 3) % 512 for i in range(ctx)]
    got, want = run.prefill(tokens[:prompt]), ref.prefill(tokens[:prompt])
    for t in tokens[prompt:]:
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
        got, want = run.decode_step(t), ref.decode_step(t)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    run.close()


@pytest.mark.parametrize("route", [None, "0", "1"])  # as the runner picks, clusters, splits
@pytest.mark.parametrize("hd,n_heads,n_kv,turns", [(64, 8, 2, (40, 20, 35, 17, 300, 30)), (64, 4, 4, (96, 17)), (128, 8, 2, (17, 31, 400, 40)), (128, 8, 1, (280, 60))])
def test_prompts_of_several_turns(backend, oracle, monkeypatch, route, hd, n_heads, n_kv, turns):
    """Short prompts after others: their queries, each with one key more than the one before, on either side of the line between the kernels."""
    if route:
        monkeypatch.setenv("YULE_CUDA_ROWS_SPLITS", route)
    cfg = ModelConfig(dim=256, n_layers=2, n_heads=n_heads, n_kv_heads=n_kv, head_dim=hd, vocab_size=512, ff_dim=512, max_seq_len=2048)
    weights = synth.synthetic_model(cfg, seed=4, std=0.08, linear=DType.Q8_0)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    for i, n in enumerate(turns):
        prompt = synth.tokens(20 + i, n, 512)
        got, want = run.prefill(prompt), ref.prefill(list(prompt))
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max(), (i, n)
    run.close()


@pytest.mark.parametrize("hd,n_heads,n_kv", [(64, 8, 2), (128, 8, 1), (128, 4, 4)])
@pytest.mark.parametrize("window,softcap", [(130, 0.0), (300, 0.0), (0, 1.5), (300, 0.7), (45, 0.7)])
def test_window_and_softcap(backend, oracle, hd, n_heads, n_kv, window, softcap):
    """Positions over one CTA, several and several clusters; window edges inside a tile.  Under a soft-cap masked positions keep a weight."""
    cfg = ModelConfig(dim=256, n_layers=2, n_heads=n_heads, n_kv_heads=n_kv, head_dim=hd, vocab_size=512, ff_dim=512, max_seq_len=2048,
                      sliding_window=window, attn_logit_softcap=softcap)
    weights = synth.synthetic_model(cfg, seed=6, std=0.15, linear=DType.Q8_0)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    tokens, at = list(synth.tokens(7, 901, 512)), 0
    for upto in (20, 46, 131, 260, 301, 431, 700, 901):
        got, want = run.prefill(tokens[at:upto]), ref.prefill(tokens[at:upto])
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max(), upto
        at = upto
    run.close()


@pytest.mark.parametrize("batch,hd,n_heads,n_kv,ctx", [(3, 64, 8, 2, 4096), (16, 128, 8, 4, 2048), (2, 128, 8, 1, 4096), (40, 64, 4, 4, 2048)])
def test_batches_at_long_contexts(backend, oracle, batch, hd, n_heads, n_kv, ctx):
    """Several clusters per KV head and sequence (the contexts are long enough for scratch): the first and the last sequence against the CPU runner."""
    cfg = ModelConfig(dim=256, n_layers=2, n_heads=n_heads, n_kv_heads=n_kv, head_dim=hd, vocab_size=512, ff_dim=512, max_seq_len=ctx)
    weights = synth.synthetic_model(cfg, seed=8, std=0.08, linear=DType.Q8_0)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), [make_oracle_model(oracle, cfg, weights) for _ in range(2)]
    steps = 520
    tokens = synth.tokens(9, batch * steps, 512).reshape(batch, steps)
    for i in range(steps):
        got = run.decode_batch(tokens[:, i])
        for b, m in zip((0, batch - 1), ref):
            want = m.decode_step(int(tokens[b, i]))
            assert np.abs(got[b] - want).max() <= 1e-4 * np.abs(want).max(), (b, i)
    run.close()
