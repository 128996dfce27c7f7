"""Row buffers of long prompts: what they hold, and prompts that run where the large ones cannot be had.  (The reference
feeds a prompt token by token and has no such buffers, yule-infer/src/gpu_runner.rs:146-160.)"""

import numpy as np
import pytest

from conftest import REL_TOL
from test_gpu_runner import guarded_rel_err
from yule_b200 import CudaB200Backend, CudaTransformerRunner, DType, ModelConfig, YuleGpuError, synth

pytestmark = pytest.mark.gpu

CFG = ModelConfig(dim=2048, n_layers=1, n_heads=16, n_kv_heads=4, head_dim=128, vocab_size=512, ff_dim=16384, max_seq_len=2304)


def free_bytes() -> int:
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.fixture(scope="module")
def weights():
    return synth.synthetic_model(CFG, seed=101, std=0.05, linear=DType.Q4_K)


def test_growth_is_bounded(weights):
    """Prompts of many lengths, each longer than the one before, hold at most twice what the longest one alone does (outgrown
    blocks of scratch stay, since captured graphs may use them)."""
    held = []
    for lengths in ([2040], range(520, 2041, 95)):
        b = CudaB200Backend(0)
        run = CudaTransformerRunner(b, CFG, weights, fused=1)
        run.prefill(synth.tokens(1, 20, CFG.vocab_size))
        before = free_bytes()
        for n in lengths:
            run.reset()
            run.prefill(synth.tokens(n, n, CFG.vocab_size))
        held.append(before - free_bytes())
        run.close()
        b.close()
    assert held[1] <= 2 * held[0], held


def test_long_prompts_without_memory_for_long_passes(backend, weights):
    """No memory for the buffers of 2048 rows: the prompts go through in passes of 512.  Every prompt takes as much memory as
    the one before, and once there is room the large buffers come back."""
    prompt = synth.tokens(2, 2040, CFG.vocab_size)
    prompts = synth.tokens(3, 6 * 300, CFG.vocab_size).reshape(6, 300)
    run = CudaTransformerRunner(backend, CFG, weights, fused=1)
    batch = CudaTransformerRunner(backend, CFG, weights, fused=1)
    want, want_batch = run.prefill(prompt), batch.generate_greedy_batch(prompts, 4)
    run.close()
    batch.close()
    run = CudaTransformerRunner(backend, CFG, weights, fused=1)
    batch = CudaTransformerRunner(backend, CFG, weights, fused=1)
    run.prefill(prompt[:600])
    run.reset()
    batch.generate_greedy_batch(prompts[:, :8], 2)
    # a row takes 4·(2 dim + 2 ff + ...) = 190 KB: 100 MB for 512, 390 MB for 2048 (600 tokens already hold 1024)
    taken = []
    for size in (1 << 34, 1 << 30, 1 << 26):
        while free_bytes() > size + (150 << 20):
            try:
                taken.append(backend.allocate(size))
            except YuleGpuError:
                break
    try:
        first = None
        for _ in range(4):
            run.reset()
            assert guarded_rel_err(run.prefill(prompt), want) <= REL_TOL
            assert np.array_equal(batch.generate_greedy_batch(prompts, 4), want_batch)
            first = free_bytes() if first is None else first
        assert first - free_bytes() < (8 << 20)
    finally:
        for h in taken:
            backend.free(h)
    run.reset()
    assert guarded_rel_err(run.prefill(prompt), want) <= REL_TOL
    run.close()
    batch.close()


def test_long_prompt_without_memory_for_the_tiled_attention(backend):
    """The tiled prompt attention writes its operands to the GEMM's scratch, which has to grow for a prompt of 30000 positions.  Without memory for that the prompt
    goes through the attention of short prompts."""
    cfg = ModelConfig(dim=512, n_layers=1, n_heads=2, n_kv_heads=1, head_dim=128, vocab_size=512, ff_dim=512, max_seq_len=30016)
    weights = synth.synthetic_model(cfg, seed=102, std=0.05, linear=DType.Q4_K)
    prompt = synth.tokens(4, 30000, cfg.vocab_size)
    own = CudaB200Backend(0)  # (a context whose scratch has not grown)
    run = CudaTransformerRunner(own, cfg, weights, fused=1)
    run.prefill(prompt[:3000])
    run.reset()
    taken = []
    for size in (1 << 34, 1 << 30, 1 << 26, 1 << 22):
        while free_bytes() > size + (16 << 20):
            try:
                taken.append(backend.allocate(size))
            except YuleGpuError:
                break
    try:
        got = run.prefill(prompt)
    finally:
        for h in taken:
            backend.free(h)
    run.reset()
    before = free_bytes()
    want = run.prefill(prompt)
    assert before - free_bytes() >= 36 << 20  # it grew only now
    assert guarded_rel_err(got, want) <= REL_TOL
    run.close()
    own.close()


@pytest.mark.parametrize("heads,kv_heads,head_dim,n", [(2, 1, 128, 56000), (4, 4, 64, 112000)])
def test_long_prompts_of_a_batch_without_memory_for_the_tiled_attention(backend, heads, kv_heads, head_dim, n):
    """The same for a batch: sequence by sequence through the attention of short prompts, the same picks."""
    cfg = ModelConfig(dim=512, n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, vocab_size=512, ff_dim=512, max_seq_len=n + 16)
    weights = synth.synthetic_model(cfg, seed=103, std=0.05, linear=DType.Q4_K)
    prompts = synth.tokens(5, 2 * n, cfg.vocab_size).reshape(2, n)
    own = CudaB200Backend(0)  # (a context whose scratch has not grown)
    run = CudaTransformerRunner(own, cfg, weights, fused=1)
    run.generate_greedy_batch(prompts[:, :3000], 1)
    taken = []
    for size in (1 << 34, 1 << 30, 1 << 26, 1 << 22):
        while free_bytes() > size + (16 << 20):
            try:
                taken.append(backend.allocate(size))
            except YuleGpuError:
                break
    try:
        run.reset_batch()
        got = run.generate_greedy_batch(prompts, 8)
        odd = run.generate_greedy_batch(prompts[:, :n // 512 * 512 - 510], 8)  # (the last pass has one token of each sequence)
    finally:
        for h in taken:
            backend.free(h)
    before = free_bytes()
    assert np.array_equal(run.generate_greedy_batch(prompts, 8), got)
    assert before - free_bytes() >= 36 << 20  # it grew only now
    assert np.array_equal(run.generate_greedy_batch(prompts[:, :n // 512 * 512 - 510], 8), odd)
    run.close()
    own.close()
