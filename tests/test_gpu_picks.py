"""Picks over a vocabulary split over a cluster of CTAs: greedy, sampled, and what a sampled run leaves behind."""

import numpy as np
import pytest

from yule_b200 import CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [3, 8, 9, 1000, 33001])
def test_pick_of_equal_logits_is_the_last(backend, vocab):
    """Every row of the output matrix the same: all logits are equal and the pick is the highest index
    (yule-infer/src/sampler.rs:150-163), wherever the vocabulary is cut."""
    cfg = ModelConfig(dim=256, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, vocab_size=vocab, ff_dim=512, max_seq_len=32)
    weights = synth.synthetic_model(cfg, seed=91, std=0.05, linear=DType.Q4_K)
    row = np.array(weights["output.weight"][0][:144])
    weights["output.weight"] = (np.tile(row, vocab), DType.Q4_K)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    assert run.generate_greedy([1, 2], 3).tolist() == [vocab - 1] * 3
    assert run.generate_greedy_batch([[1, 2], [2, 0]], 3).tolist() == [[vocab - 1] * 3] * 2
    run.close()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 8191, 230000])
def test_sampler_over_a_cut_vocabulary(backend, oracle, n):
    """Vocabularies smaller than the cluster, at its edges, and too large for its shared memory (slices in global
    memory); ties at the top-p boundary that are cut in index order across the CTAs."""
    logits = (4.0 * synth.normal(300 + n, n)).astype(np.float32)
    logits[n // 3:] = np.round(logits[n // 3:])  # many equal values
    lh = backend.upload(logits)
    kw = dict(temperature=0.8, top_p=0.7, top_k=0 if n < 100 else 50, repetition_penalty=1.0, min_p=0.0)
    for r in (0.013, 0.31, 0.62, 0.93):
        near = {oracle.sample(logits, float(r + d), **kw) for d in (-5e-5, 0.0, 5e-5)}
        if len(near) == 1:
            assert backend.sample(lh, n, r, **kw) == near.pop()
    backend.free(lh)


def test_filtered_tokens_are_never_picked(backend):
    """Random values at and around the mass that lies before each run of 32 tokens (what a warp adds up): runs begin and end with
    tokens that min-p removes, so a pick must be one of the tokens between."""
    n = 8192
    logits = synth.normal(310, n).reshape(-1, 32)
    logits[:, :8] = logits[:, 24:] = -30.0
    lh = backend.upload(logits.astype(np.float32).reshape(-1))
    kept = np.exp(logits.astype(np.float64))
    kept[:, :8] = kept[:, 24:] = 0
    edges = np.cumsum(kept.sum(1) / kept.sum())[:-1:3].astype(np.float32)
    kw = dict(temperature=1.0, top_p=1.0, top_k=0, repetition_penalty=1.0, min_p=1e-6)
    for edge in edges:
        for step in range(-4, 5):
            r = np.uint32(int(edge.view(np.uint32)) + step).view(np.float32)
            assert 8 <= backend.sample(lh, n, float(r), **kw) % 32 < 24, (float(r), step)
    backend.free(lh)


def test_sampled_stream_continues_greedily(backend):
    """A sampled run leaves the runner where feeding its tokens would have left it."""
    cfg = ModelConfig(dim=512, n_layers=2, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=700, ff_dim=768, max_seq_len=128)
    weights = synth.synthetic_model(cfg, seed=95, std=0.05, linear=DType.Q8_0)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    prompt = synth.tokens(96, 12, cfg.vocab_size)
    picks = run.generate_sampled(prompt, 9, seed=5)
    more = run.generate_greedy([], 5)
    run.reset()
    assert np.array_equal(run.generate_sampled(prompt, 9, seed=5), picks)
    run.reset()
    assert np.array_equal(run.generate_greedy(np.concatenate([prompt, picks]), 5), more)
    run.close()
