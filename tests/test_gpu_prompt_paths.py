"""Prompts that share their passes over the weights: the tiled causal attention (128 query rows per CTA against 64-position
tiles of the fp32 cache) and prompts of a whole batch.  Oracle: the CPU runner restated (yule-infer/src/model_runner.rs:533-1036), which feeds one token at a time."""

import numpy as np
import pytest

from conftest import REL_TOL
from test_gpu_runner import guarded_rel_err, make_oracle_model
from yule_b200 import CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 1, 64), (8, 4, 64), (4, 4, 64), (8, 1, 128), (8, 2, 128), (4, 4, 128)])
@pytest.mark.parametrize("n", [17, 65, 129, 200, 577])
def test_tiled_prompt_attention(backend, oracle, heads, kv_heads, head_dim, n):
    """One query tile and several, one K / V tile, its edge and several, then a second prompt that starts inside a tile.  (With so few
    heads only more than 512 tokens go through the tiled kernel; the others stay below its line.)"""
    cfg = ModelConfig(dim=512, n_layers=1, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=300, ff_dim=512,
                      max_seq_len=700)
    weights = synth.synthetic_model(cfg, seed=60 + n, std=0.06, linear=DType.Q4_K)
    ref = make_oracle_model(oracle, cfg, weights)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    for part, m in enumerate((n, 70)):
        prompt = synth.tokens(5 + part, m, cfg.vocab_size)
        assert guarded_rel_err(run.prefill(prompt), ref.prefill(prompt)) <= REL_TOL
    assert guarded_rel_err(run.decode_step(7), ref.decode_step(7)) <= REL_TOL
    run.close()


def test_tiled_prompt_attention_large_and_small_values(backend, oracle):
    """Values far outside fp16's range and far below its normal numbers: every K / V tile has its own power of two."""
    cfg = ModelConfig(dim=256, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, vocab_size=300, ff_dim=512, max_seq_len=160)
    for factor in (3e4, 2e-3):
        weights = synth.synthetic_model(cfg, seed=70, std=0.06, linear=DType.Q4_K)
        data, dt = weights["blk.0.attn_v.weight"]
        blocks = np.array(data).reshape(-1, 144).copy()
        d = blocks[:, :4].copy().view(np.float16).astype(np.float32) * np.float32(factor)  # d and dmin
        blocks[:, :4] = d.astype(np.float16).view(np.uint8)
        weights["blk.0.attn_v.weight"] = (blocks.reshape(-1), dt)
        ref = make_oracle_model(oracle, cfg, weights)
        run = CudaTransformerRunner(backend, cfg, weights, fused=1)
        prompt = synth.tokens(8, 130, cfg.vocab_size)
        assert guarded_rel_err(run.prefill(prompt), ref.prefill(prompt)) <= REL_TOL
        run.close()


def unit_rows(columns, dim, factor=1.0):
    """Q8_0 matrix whose row r is `factor` times the unit vector `columns[r]`."""
    blocks = np.zeros((len(columns), dim // 32, 34), np.uint8)
    for r, c in enumerate(columns):
        blocks[r, c // 32, :2] = np.array([factor], np.float16).view(np.uint8)
        blocks[r, c // 32, 2 + c % 32] = 1
    return blocks.reshape(-1), DType.Q8_0


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 64), (4, 1, 128)])
def test_prompt_attention_error(backend, heads, kv_heads, head_dim):
    """The tiled attention against 64 bits.  Matrices of unit vectors make its operands known: the first layer's caches hold them
    (a query is -4 times the K row of its position), and the second layer's V rows are its normalised output, 32 times as large as the
    hidden state it is added to.  The bound: the scores are about N(0, 4^2), and rounding one of 8 to 16 to 24 bits alone moves its
    probability by up to 8 units of 2^-24.  (This kernel 3.4 and 3.7 units; with all MMAs of a sum on one accumulator, which
    truncates, 11 and 18.)"""
    n, dim, kv = 700, 512, kv_heads * head_dim
    cfg = ModelConfig(dim=dim, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=800, ff_dim=512, max_seq_len=768)
    weights = synth.synthetic_model(cfg, seed=92, std=0.06, linear=DType.Q8_0, token_embd=DType.Q8_0)
    group = heads // kv_heads
    for layer in range(2):
        name = f"blk.{layer}."
        weights[name + "attn_q.weight"] = unit_rows([r // (group * head_dim) * head_dim + r % head_dim for r in range(dim)], dim, -4.0)
        weights[name + "attn_k.weight"] = unit_rows(range(kv), dim)
        weights[name + "attn_v.weight"] = unit_rows(range(dim - kv, dim) if layer == 0 else [r // head_dim * group * head_dim + r % head_dim for r in range(kv)], dim)
        weights[name + "attn_output.weight"] = unit_rows(range(dim), dim, 32.0)
        weights[name + "ffn_down.weight"] = (np.zeros(dim * cfg.ff_dim // 32 * 34, np.uint8), DType.Q8_0)
        for norm in ("attn_norm", "ffn_norm"):
            weights[name + norm + ".weight"] = (np.ones(dim, np.float32).view(np.uint8), DType.F32)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    prompt = synth.tokens(93, n, cfg.vocab_size)
    run.prefill(prompt)
    m = n - 1  # the last token goes through the token step
    k, v, out = (backend.download(run.buffer(which, layer), n * kv).astype(np.float64).reshape(n, kv_heads, head_dim)[:m]
                 for which, layer in (("k_cache", 0), ("v_cache", 0), ("v_cache", 1)))
    run.close()
    embd = np.array(weights["token_embd.weight"][0]).reshape(cfg.vocab_size, dim // 32, 34)
    x = (embd[:, :, :2].copy().view(np.float16).astype(np.float64) * embd[:, :, 2:].copy().view(np.int8)).reshape(cfg.vocab_size, dim)[prompt[:m]]
    s = np.einsum("ihd,jhd->hij", -4 * k, k) / np.sqrt(head_dim)
    s[:, np.arange(m)[:, None] < np.arange(m)] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    att = np.einsum("hij,jhd->ihd", p / p.sum(-1, keepdims=True), v)
    hidden = x + 32 * np.repeat(att, group, axis=1).reshape(m, dim)
    normed = hidden / np.sqrt((hidden ** 2).mean(-1, keepdims=True) + cfg.norm_eps)
    want = normed.reshape(m, kv_heads, group, head_dim)[:, :, 0]
    error = np.linalg.norm(out - want) / np.linalg.norm(want)
    assert error <= 8 * 2.0 ** -24, error


@pytest.mark.parametrize("offset", [1000, -1000, 2100, 4200, -4200, 8000])
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 2, 64), (4, 1, 128)])
def test_prompt_attention_with_large_scores(backend, heads, kv_heads, head_dim, offset):
    """Scores of N(0, 1) beside a constant in the thousands, the same for all positions, which cancels in the soft-max.  As in test_prompt_attention_error, but the
    hidden states are +1 and -1, so that their norm is the same for all tokens, and one channel of a head is +1 in all of them, has a large weight in the norm and belongs
    to the pair that RoPE all but leaves alone.  The bound: a score rounded to 24 bits moves its probability by up to |offset| units of 2^-24, once where it is added up and
    once where it is scaled; 8 units as without the constant.  (2 to 6 units where every position prefers itself, 26 to 104 where it prefers all others.)"""
    n, dim, kv = 700, 512, kv_heads * head_dim
    cfg = ModelConfig(dim=dim, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=800, ff_dim=512, max_seq_len=768, rope_freq_base=1e30)
    weights = synth.synthetic_model(cfg, seed=94, std=0.06, linear=DType.Q8_0, token_embd=DType.Q8_0)
    channels = np.arange(kv_heads) * head_dim + head_dim - 1
    x = np.where(np.random.default_rng(95).random((cfg.vocab_size, dim)) < 0.5, -1, 1).astype(np.int8)
    x[:, channels] = 1
    embd = np.zeros((cfg.vocab_size, dim // 32, 34), np.uint8)
    embd[:, :, :2] = np.array([1.0], np.float16).view(np.uint8)
    embd[:, :, 2:] = x.view(np.uint8).reshape(cfg.vocab_size, dim // 32, 32)
    weights["token_embd.weight"] = (embd.reshape(-1), DType.Q8_0)
    group, sign = heads // kv_heads, np.sign(offset)
    for layer in range(2):
        name = f"blk.{layer}."
        weights[name + "attn_q.weight"] = unit_rows([r // (group * head_dim) * head_dim + r % head_dim for r in range(dim)], dim, sign)
        weights[name + "attn_k.weight"] = unit_rows(range(kv), dim)
        weights[name + "attn_v.weight"] = unit_rows(range(dim - kv, dim) if layer == 0 else [r // head_dim * group * head_dim + r % head_dim for r in range(kv)], dim)
        weights[name + "attn_output.weight"] = unit_rows(range(dim), dim, 32.0)
        weights[name + "ffn_down.weight"] = (np.zeros(dim * cfg.ff_dim // 32 * 34, np.uint8), DType.Q8_0)
        for norm in ("attn_norm", "ffn_norm"):
            w = np.ones(dim, np.float32)
            if norm == "attn_norm" and layer == 0:
                w[channels] = np.sqrt(abs(offset) * np.sqrt(head_dim))
            weights[name + norm + ".weight"] = (w.view(np.uint8), DType.F32)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    prompt = synth.tokens(96, n, cfg.vocab_size)
    run.prefill(prompt)
    m = n - 1  # the last token goes through the token step
    k, v, out = (backend.download(run.buffer(which, layer), n * kv).astype(np.float64).reshape(n, kv_heads, head_dim)[:m]
                 for which, layer in (("k_cache", 0), ("v_cache", 0), ("v_cache", 1)))
    run.close()
    s = np.einsum("ihd,jhd->hij", sign * k, k) / np.sqrt(head_dim)
    assert abs(s - offset).max() < 0.02 * abs(offset)
    s[:, np.arange(m)[:, None] < np.arange(m)] = -np.inf
    p = np.exp(s - s.max(-1, keepdims=True))
    att = np.einsum("hij,jhd->ihd", p / p.sum(-1, keepdims=True), v)
    hidden = x[prompt[:m]].astype(np.float64) + 32 * np.repeat(att, group, axis=1).reshape(m, dim)
    normed = hidden / np.sqrt((hidden ** 2).mean(-1, keepdims=True) + cfg.norm_eps)
    want = normed.reshape(m, kv_heads, group, head_dim)[:, :, 0]
    error = np.linalg.norm(out - want) / np.linalg.norm(want)
    assert error <= (8 + 2 * abs(offset)) * 2.0 ** -24, error


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(8, 1, 64), (8, 2, 128)])
@pytest.mark.parametrize("size", ["infinite", "huge"])
def test_later_tokens_do_not_reach_earlier_ones(backend, oracle, heads, kv_heads, head_dim, size):
    """A token whose K and V rows are not finite, or 10^24 times as large as the others', shares a K / V tile with tokens before
    it: what those compute (the K rows of the second layer) is what they compute without it."""
    n, at, odd = 600, 550, 299  # more than 512 tokens always go through the tiled kernel
    cfg = ModelConfig(dim=512, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=300, ff_dim=512,
                      max_seq_len=640)
    weights = synth.synthetic_model(cfg, seed=90, std=0.06, linear=DType.Q4_K, token_embd=DType.Q8_0)
    embd = np.array(weights["token_embd.weight"][0]).reshape(cfg.vocab_size, cfg.dim // 32, 34).copy()
    if size == "infinite":
        embd[odd, :, :2] = np.full(1, np.inf, np.float16).view(np.uint8)
    else:  # one element of the hidden state that only this token has, and a large weight for it in the first norm
        embd[:, 0, 2] = 0
        embd[odd, 0, 2] = 100
        norm = np.ones(cfg.dim, np.float32)
        norm[0] = 1e25
        weights["blk.0.attn_norm.weight"] = (norm.view(np.uint8), DType.F32)
    weights["token_embd.weight"] = (embd.reshape(-1), DType.Q8_0)
    prompt = synth.tokens(91, n, odd)
    prompt[at] = odd
    ref = make_oracle_model(oracle, cfg, weights)
    ref.prefill(prompt[:at])
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    run.prefill(prompt)
    kv = cfg.n_kv_heads * cfg.head_dim
    rows = backend.download(run.buffer("k_cache", 1), n * kv).reshape(n, kv)
    assert guarded_rel_err(rows[:at].reshape(-1), np.asarray(ref.k_cache(1, at)).reshape(-1)) <= REL_TOL
    assert size == "huge" or np.isnan(rows[at:]).all()
    run.close()


@pytest.mark.parametrize("batch,n_prompt", [(3, 5), (2, 70), (9, 33), (33, 65)])
def test_batch_prompts_in_passes(backend, batch, n_prompt):
    """Prompts of all sequences in shared passes (more rows than one pass takes in the last case) against the same
    sequences one by one."""
    cfg = ModelConfig(dim=512, n_layers=2, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=700, ff_dim=768, max_seq_len=128)
    weights = synth.synthetic_model(cfg, seed=81, std=0.05, linear=DType.Q4_K, ffn_down=DType.Q6_K, output=DType.Q6_K)
    prompts = synth.tokens(82, batch * n_prompt, cfg.vocab_size).reshape(batch, n_prompt)
    run = CudaTransformerRunner(backend, cfg, weights, fused=1)
    got = run.generate_greedy_batch(prompts, 6)
    again = run.generate_greedy_batch(prompts, 6)
    assert np.array_equal(got, again)
    single = CudaTransformerRunner(backend, cfg, weights, fused=1)
    for b in {0, batch // 2, batch - 1}:
        single.reset()
        assert np.array_equal(got[b], single.generate_greedy(prompts[b], 6)), f"sequence {b}"
    # a larger pass replaces the row buffers of the runner: the captured step must follow
    longer = synth.tokens(83, batch * 100, cfg.vocab_size).reshape(batch, 100)
    run.generate_greedy_batch(longer, 2)
    assert np.array_equal(run.generate_greedy_batch(prompts, 6), got)
    single.close()
    run.close()
