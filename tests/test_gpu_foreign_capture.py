"""Calls beside another stream of the process whose capture forbids allocations to everyone."""

import ctypes

import pytest

from conftest import guarded_rel_err, REL_TOL
from yule_b200 import CudaB200Backend, DType, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,batch", [(DType.Q4_0, 24), (DType.Q5_K, 20), (DType.Q8_0, 17), (DType.Q6_K, 32), (DType.Q4_K, 70)])
def test_scratch_of_the_gemm(oracle, dtype, batch):
    """The first GEMM of a context allocates.  The call goes through and the capture goes on."""
    n_rows, n_cols = 4224, 4096
    b = CudaB200Backend(0)  # (a context whose scratch has not grown)
    w, x = synth.random_quantized(dtype, 61, n_rows * n_cols), synth.normal(62, batch * n_cols)
    wh, xh, oh = b.upload(w), b.upload(x), b.allocate(batch * n_rows * 4)
    b.prepare_weights(wh, dtype, n_rows, n_cols)
    b.synchronize()
    driver, stream, graph = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(), ctypes.c_void_p()
    assert driver.cuStreamCreate(ctypes.byref(stream), 1) == 0
    assert driver.cuStreamBeginCapture_v2(stream, 0) == 0
    try:
        b.quantized_matmul_batched(wh, xh, oh, n_rows, n_cols, dtype, batch)
    finally:
        ended = driver.cuStreamEndCapture(stream, ctypes.byref(graph))
        driver.cuStreamDestroy_v2(stream)
    assert ended == 0 and driver.cuGraphDestroy(graph) == 0
    y = b.download(oh, batch * n_rows).reshape(batch, n_rows)
    for i in (0, batch - 1):
        assert guarded_rel_err(y[i], oracle.qmv(int(dtype), w, x[i * n_cols:(i + 1) * n_cols], n_rows, n_cols)) <= REL_TOL
    b.close()
