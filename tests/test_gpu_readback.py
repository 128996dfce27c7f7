"""Small results to the host (csrc/readback.cu): sizes around its vector width, its CTAs' shares and the line to the copy engine, into
pageable, unaligned and pinned memory; behind a matvec as its dependent launch; from several threads."""

import ctypes
import mmap
import threading

import numpy as np
import pytest
import torch

from yule_b200 import DType, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4095, 4096, 4097, 64 * 4096 + 5, (1 << 20) - 1, 1 << 20, (1 << 20) + 1])
def test_sizes_and_destinations(backend, n):
    data = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    h = backend.upload(data)
    pinned = torch.zeros(n + 64, dtype=torch.uint8).pin_memory().numpy()
    for dst in (np.zeros(n, np.uint8), np.zeros(n + 8, np.uint8)[3:3 + n], pinned[:n], pinned[16:16 + n], pinned[5:5 + n]):
        dst[:] = 0
        backend.copy_from_device(h, dst)
        assert np.array_equal(dst, data)
    assert pinned[16 + n:].max(initial=0) == 0  # nothing behind the end
    backend.free(h)


def test_behind_a_matvec_and_from_threads(backend, oracle):
    rows, cols = 1000, 2048
    w, x = synth.random_quantized(DType.Q4_K, 5, rows * cols), synth.normal(6, cols)
    wh, xh = backend.upload(w), backend.upload(x)
    outs = [backend.allocate(rows * 4) for _ in range(4)]
    ref = oracle.qmv(int(DType.Q4_K), w, x, rows, cols)
    for _ in range(20):
        backend.quantized_matmul(wh, xh, outs[0], rows, cols, DType.Q4_K)
        assert np.abs(backend.download(outs[0], rows) - ref).max() <= 1e-5 * np.abs(ref).max()
    for o in outs[1:]:
        backend.quantized_matmul(wh, xh, o, rows, cols, DType.Q4_K)
    good = [0] * 4

    def read(i):
        for _ in range(200):
            y = np.zeros(rows, np.float32)
            backend.copy_from_device(outs[i], y)
            good[i] += int(np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max())

    threads = [threading.Thread(target=read, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert good == [200] * 4


def test_every_byte_is_there_when_the_call_returns(backend):
    """The last CTA's fence has to cover the stores of the others: the destination is looked at at once, each time with other contents."""
    n = 1 << 20
    a = np.random.default_rng(1).integers(0, 256, n, dtype=np.uint8)
    both = a, ~a
    handles = [backend.upload(x) for x in both]
    pinned = torch.zeros(n, dtype=torch.uint8).pin_memory().numpy()
    for size in (5000, 70000, n):
        for i in range(200):
            backend.copy_from_device(handles[i & 1], pinned[:size])
            assert np.array_equal(pinned[:size], both[i & 1][:size])
    for h in handles:
        backend.free(h)


@pytest.mark.parametrize("registered", [
    [(0, 4096, 3), (12288, 4096, 3)],   # the ends of the destination, not its middle: a kernel's stores to the middle would fault
    [(0, 8192, 3)],                     # its beginning
    [(8192, 8192, 3)],                  # its end
    [(0, 16384, 3)],                    # all of it
    [(0, 16384, 8 | 3)],                # all of it, read-only for the device
])
def test_destinations_that_a_kernel_may_not_store_to(backend, registered):
    """Memory that is registered in part, or read-only, gets its bytes from the host."""
    cuda = ctypes.CDLL("libcuda.so.1")
    data = np.random.default_rng(2).integers(0, 256, 16384, dtype=np.uint8)
    h, area = backend.upload(data), mmap.mmap(-1, 16384)
    dst = np.frombuffer(area, np.uint8)
    base = dst.ctypes.data
    for at, size, flags in registered:
        assert cuda.cuMemHostRegister_v2(ctypes.c_void_p(base + at), ctypes.c_size_t(size), flags) == 0
    try:
        for lo, hi in ((0, 16384), (16, 16384), (0, 16000)):
            dst[:] = 0
            backend.copy_from_device(h, dst[lo:hi])
            assert np.array_equal(dst[lo:hi], data[:hi - lo])
    finally:
        for at, _, _ in registered:
            cuda.cuMemHostUnregister(ctypes.c_void_p(base + at))
        backend.free(h)


def test_managed_memory(backend):
    cuda = ctypes.CDLL("libcuda.so.1")
    data = np.random.default_rng(3).integers(0, 256, 10000, dtype=np.uint8)
    h, ptr = backend.upload(data), ctypes.c_ulonglong()
    assert cuda.cuMemAllocManaged(ctypes.byref(ptr), ctypes.c_size_t(10000), 1) == 0
    dst = np.frombuffer((ctypes.c_ubyte * 10000).from_address(ptr.value), np.uint8)
    backend.copy_from_device(h, dst)
    assert np.array_equal(dst, data)
    cuda.cuMemFree_v2(ptr)
    backend.free(h)


def test_logits_beyond_the_line_to_the_copy_engine(backend, oracle):
    """262144 logits are 1 MiB."""
    from test_gpu_runner import make_oracle_model
    from yule_b200 import CudaTransformerRunner, ModelConfig
    cfg = ModelConfig(dim=256, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=64, vocab_size=262400, ff_dim=256, max_seq_len=16)
    weights = synth.synthetic_model(cfg, seed=3, std=0.05, linear=DType.Q8_0)
    run, ref = CudaTransformerRunner(backend, cfg, weights, fused=1), make_oracle_model(oracle, cfg, weights)
    got, want = run.prefill([1, 2]), ref.prefill([1, 2])
    for t in (262399, 5):
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
        got, want = run.decode_step(t), ref.decode_step(t)
    assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()
    run.close()
