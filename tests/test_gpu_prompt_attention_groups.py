"""The prompt attention (csrc/attn_prefill.cu) where its scratch holds the operands of some KV heads at a time only."""

import numpy as np
import pytest

from yule_b200 import CudaB200Backend, CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim,n", [(8, 8, 128, 4300), (16, 8, 64, 7700)])
def test_heads_in_groups(heads, kv_heads, head_dim, n):
    """80 (40) KB per KV head and 64 positions: more than the scratch of a fresh context holds, less than that of one that has run a wide GEMM.  The same bits."""
    cfg = ModelConfig(dim=1024, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=400, ff_dim=512, max_seq_len=n + 8)
    weights = synth.synthetic_model(cfg, seed=31, std=0.05, linear=DType.Q4_K)
    prompt = synth.tokens(32, n, cfg.vocab_size)
    got = []
    for wide in (False, True):
        b = CudaB200Backend(0)
        if wide:
            w, x, y = b.upload(synth.random_blocks(DType.Q4_K, 1, 112)), b.allocate(400 * 28672 * 4), b.allocate(400 * 4)
            b.quantized_matmul_batched(w, x, y, 1, 28672, DType.Q4_K, 400)
        run = CudaTransformerRunner(b, cfg, weights, fused=1)
        logits = run.prefill(prompt)
        got.append((logits, b.download(run.buffer("v_cache", 1), n * kv_heads * head_dim)))
        run.close()
        b.close()
    for a, c in zip(*got):
        assert np.isfinite(a).all() and np.array_equal(a.view(np.uint32), c.view(np.uint32))
