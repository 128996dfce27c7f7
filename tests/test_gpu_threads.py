"""Entry points of one context from several threads (include/yule_cuda.h: all are thread-safe): every thread gets the bits that it gets alone."""

from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from test_gpu_op_chain import build, play, steps
from yule_b200 import CudaTransformerRunner, DType, ModelConfig, synth

pytestmark = pytest.mark.gpu


def together(jobs):
    with ThreadPoolExecutor(len(jobs)) as pool:
        return [f.result() for f in [pool.submit(j) for j in jobs]]


def same(got, want):
    assert len(got) == len(want)
    return all(np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32)) for a, b in zip(got, want))


@pytest.mark.parametrize("threads", [2, 5])
def test_chains_of_ops(backend, threads):
    """The chain of dependent launches is the context's: each thread's outputs have to stay in its list, which has to stay within its bounds."""
    todo = [steps(np.random.default_rng(300 + i), 300) for i in range(threads)]
    want = [play(backend, build(backend), t, False) for t in todo]
    for _ in range(3):
        got = together([lambda t=t: play(backend, build(backend), t, False) for t in todo])
        assert all(same(g, w) for g, w in zip(got, want))


def gemms(backend, dtype, batch, n_rows, n_cols, times=25):
    w, x = synth.random_quantized(dtype, 7, n_rows * n_cols), synth.normal(8 + batch, batch * n_cols)
    wh, xh, oh = backend.upload(w), backend.upload(x), backend.allocate(batch * n_rows * 4)
    backend.prepare_weights(wh, dtype, n_rows, n_cols)

    def go():
        out = []
        for _ in range(times):
            backend.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
            out.append(backend.download(oh, batch * n_rows))
        return out
    return go, (wh, xh, oh)


def test_gemms_and_a_prompt(backend):
    """The re-layout and the GEMM behind it, and the launches of a prompt's pass, hand the context's scratch on: no other thread's come in between."""
    cfg = ModelConfig(dim=512, n_layers=3, n_heads=8, n_kv_heads=2, head_dim=64, vocab_size=300, ff_dim=1024, max_seq_len=700)
    run = CudaTransformerRunner(backend, cfg, synth.synthetic_model(cfg, seed=9, std=0.05, linear=DType.Q4_K), fused=1)
    prompt = synth.tokens(10, 600, cfg.vocab_size)

    def prompts():
        out = []
        for _ in range(12):
            run.reset()
            out.append(run.prefill(prompt))
        return out
    made = [gemms(backend, *a) for a in ((DType.Q4_K, 100, 512, 2048), (DType.Q8_0, 40, 1024, 1024), (DType.Q6_K, 33, 300, 4096), (DType.Q5_K, 50, 256, 512))]
    jobs = [go for go, _ in made] + [prompts]
    want = [j() for j in jobs]
    for _ in range(2):
        assert all(same(g, w) for g, w in zip(together(jobs), want))
    run.close()
    for _, handles in made:
        for h in handles:
            backend.free(h)


def test_samples(backend):
    logits = [backend.upload(synth.normal(20 + i, 32000) * 3) for i in range(4)]
    jobs = [lambda h=h: [backend.sample(h, 32000, (k + 0.5) / 60) for k in range(60)] for h in logits]
    want = [j() for j in jobs]
    assert together(jobs) == want
    for h in logits:
        backend.free(h)
