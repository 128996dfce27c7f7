"""Ops of a forward pass as a chain of programmatic dependent launches: the same bits as with a wait after every call, whatever reads what another has
just written (inputs, weights, caches), with more outputs than the list of the chain holds, and in a captured graph."""

import numpy as np
import pytest

from yule_b200 import DType, synth

pytestmark = pytest.mark.gpu

DIM, HD, HEADS, KV = 512, 64, 8, 2


def build(backend, n_vectors=40):
    h = {"v": [backend.upload(synth.normal(10 + i, DIM)) for i in range(n_vectors)],
         "w": [backend.upload(synth.random_quantized(t, 60 + i, DIM * DIM)) for i, t in enumerate((DType.Q4_K, DType.Q8_0, DType.Q6_K, DType.Q4_K))],
         "spare": backend.upload(synth.random_quantized(DType.Q4_K, 99, DIM * DIM)), "norm": backend.upload(np.ones(DIM, np.float32)),
         "cache": [backend.upload(synth.normal(200 + i, 40 * KV * HD)) for i in range(2)]}
    backend.prepare_weights(h["w"][2], DType.Q6_K, DIM, DIM)
    return h


def steps(rng, n):
    """Random calls over few vectors, so that most read what one of the last few wrote."""
    kinds = ["norm", "mat", "mat", "mat", "add", "mul", "silu", "rope", "append", "attention", "reload", "batch"]
    return [(rng.choice(kinds), *rng.integers(0, 40, 4)) for _ in range(n)]


def play(backend, h, todo, wait):
    for kind, a, b, c, d in todo:
        v = h["v"]
        few = lambda i: v[i % 6]  # noqa: E731
        if kind == "norm":
            backend.rms_norm(few(a), h["norm"], few(b), DIM, 1e-5)
        elif kind == "mat":
            t = (DType.Q4_K, DType.Q8_0, DType.Q6_K, DType.Q4_K)[c % 4]
            backend.quantized_matmul(h["w"][c % 4], few(a), v[d] if d > 20 else few(a + 1 + b % 5), DIM, DIM, t)
        elif kind == "add":
            backend.add(few(a), v[b], few(c), DIM)
        elif kind == "mul":
            backend.element_mul(few(a), few(b), few(c), DIM)
        elif kind == "silu":
            backend.silu(few(a), few(a + 1 + b % 5), DIM)
        elif kind == "rope":
            backend.rope(few(a), few(a + 1 + b % 5), int(c), HD, 10000.0, HEADS, KV)
        elif kind == "append":
            backend.copy_buffer_offset(few(a), h["cache"][b % 2], 0, int(c) * KV * HD * 4, KV * HD * 4)
        elif kind == "attention":
            backend.multihead_attention(few(a), h["cache"][0], h["cache"][1], few(a + 1 + b % 5), HD, 1 + int(c), HEADS, KV, KV * HD)
        elif kind == "reload":  # part of a matrix overwritten by a copy that belongs to the chain: what reads it has to wait
            backend.copy_buffer_offset(h["spare"], h["w"][3], int(a) * 144, int(b) * 144, 144 * 8)
        else:
            backend.quantized_matmul_batched(h["w"][0], few(a), v[10 + d % 3], DIM // 2, DIM // 2, DType.Q4_K, 2, DIM // 2, DIM // 2)
        # values stay in range: a vector that has been written is normalised now and then
        if d % 4 == 0:
            backend.rms_norm(few(c), h["norm"], few(c), DIM, 1e-5)
        if wait:
            backend.synchronize()
    out = [backend.download(x, DIM) for x in h["v"]] + [backend.download(x, 40 * KV * HD) for x in h["cache"]]
    for x in h["v"] + h["w"] + h["cache"] + [h["spare"], h["norm"]]:
        backend.free(x)
    return out


@pytest.mark.parametrize("seed", range(6))
def test_same_bits_as_with_a_wait_after_every_call(backend, seed):
    todo = steps(np.random.default_rng(seed), 400)
    got, want = (play(backend, build(backend), todo, wait) for wait in (False, True))
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_attention_on_the_built_in_scratch(backend):
    """It ends the chain: the matvec of what it has written waits for it.  (Some 20 us of attention, of which the matvec's start is 2.)"""
    seq = 6000
    q, x, y = backend.upload(synth.normal(1, DIM)), backend.upload(synth.normal(2, DIM)), backend.allocate(DIM * 4)
    k, v = (backend.upload(synth.normal(3 + i, seq * KV * HD)) for i in range(2))
    w = backend.upload(synth.random_quantized(DType.Q4_K, 5, DIM * DIM))
    got = []
    for wait in (False, True) * 20:
        backend.copy_to_device(synth.normal(100 + len(got) // 2, DIM), q)
        backend.rope(q, x, 7, HD, 10000.0, HEADS, HEADS)
        backend.multihead_attention_static(q, k, v, x, HD, seq, HEADS, KV, KV * HD)
        if wait:
            backend.synchronize()
        backend.quantized_matmul(w, x, y, DIM, DIM, DType.Q4_K)
        got.append(backend.download(y, DIM))
    for a, b in zip(got[::2], got[1::2]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    for h in (q, x, y, k, v, w):
        backend.free(h)


def test_captured(backend):
    todo = steps(np.random.default_rng(77), 120)
    h, other = build(backend), build(backend)
    backend.graph_begin()
    for step in todo:
        play_one(backend, h, step)
    backend.graph_launch(backend.graph_end())
    backend.synchronize()
    for step in todo:
        play_one(backend, other, step)
        backend.synchronize()
    for a, b in zip(h["v"], other["v"]):
        assert np.array_equal(backend.download(a, DIM).view(np.uint32), backend.download(b, DIM).view(np.uint32))


def play_one(backend, h, step):
    kind, a, b, c, d = step
    few = lambda i: h["v"][i % 6]  # noqa: E731
    if kind == "mat":
        backend.quantized_matmul(h["w"][0], few(a), few(a + 1 + b % 5), DIM, DIM, DType.Q4_K)
    elif kind == "append":
        backend.copy_buffer_offset(few(a), h["cache"][b % 2], 0, int(c) * KV * HD * 4, KV * HD * 4)
    elif kind == "add":
        backend.add(few(a), h["v"][b], few(c), DIM)
    else:
        backend.rms_norm(few(a), h["norm"], few(b), DIM, 1e-5)


@pytest.mark.parametrize("src,dst,size", [(0, 0, 16), (0, 16, 4096), (16, 0, 262144), (0, 0, 262144 + 16), (4, 8, 100), (0, 4, 32), (8, 8, 24), (0, 0, 1)])
def test_copies_of_every_alignment(backend, src, dst, size):
    """Multiples of 16 up to 256 KB by a kernel, everything else by the copy engine; the bytes around them stay."""
    a, b = np.arange(300000, dtype=np.uint32).view(np.uint8)[:600000].copy(), np.full(600000, 7, np.uint8)
    ha, hb = backend.upload(a), backend.upload(b)
    backend.copy_buffer_offset(ha, hb, src, dst, size)
    want = b.copy()
    want[dst:dst + size] = a[src:src + size]
    got = np.empty(600000, np.uint8)
    backend.copy_from_device(hb, got)
    assert np.array_equal(got, want)
    for h in (ha, hb):
        backend.free(h)


@pytest.mark.parametrize("n", [1, 255, 257, 148 * 8 * 256, 148 * 8 * 256 + 1, 304127, 304128, 304129, 1 << 20, (1 << 20) + 769])
def test_add(backend, n):
    """One element a thread and four; into a buffer of its own and into an operand's; what lies behind stays."""
    a, b = (synth.normal(seed, n + 40) for seed in (7, 8))
    ha, hb, ho = backend.upload(a), backend.upload(b), backend.upload(np.full(n + 40, 3.0, np.float32))
    backend.add(ha, hb, ho, n)
    backend.add(ha, hb, hb, n)
    assert np.array_equal(backend.download(ho, n + 40), np.concatenate([a[:n] + b[:n], np.full(40, 3.0, np.float32)]))
    assert np.array_equal(backend.download(hb, n + 40), np.concatenate([a[:n] + b[:n], b[n:]]))
    for h in (ha, hb, ho):
        backend.free(h)


@pytest.mark.parametrize("n", [1, 4096, 65536, 65537, 1 << 20])
def test_a_pinned_source_may_be_overwritten_when_the_call_returns(backend, n):
    """Up to 64 KB it goes the way of a pageable one, beyond that the call waits."""
    import torch
    host = torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()
    h, got = backend.allocate(n), np.empty(n, np.uint8)
    for value in range(1, 20):
        host[:] = value
        backend.copy_to_device(host, h)
        host[:] = 200
        if value % 6 == 0:
            backend.copy_from_device(h, got)
            assert np.all(got == value)
    backend.free(h)
