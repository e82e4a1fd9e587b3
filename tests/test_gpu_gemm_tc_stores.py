"""The tensor-core GEMM's two ways of storing C (csrc/gemm_tc.cu): four columns at a
time where rows, pitch and base are whole float4s, one at a time otherwise, at
column counts around a load of 16 and a tile of 128, one and two K slices, and with
the elements of C's pitch beyond N left alone.  Within 1e-4 of the largest FP64 product of the same
BF16 operands (FP32 accumulation), the bound of the other GEMM test."""
import ctypes

import numpy as np
import pytest

from test_gpu_gemm_tc import bf16

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,pad,shift", [
    (33, 4, 4, 0, 0), (33, 16, 64, 4, 0), (130, 20, 68, 0, 0), (64, 124, 128, 8, 0), (129, 132, 64, 0, 0),
    (33, 4, 4, 1, 0), (33, 16, 64, 0, 1), (130, 19, 68, 1, 0), (65, 132, 132, 4, 3), (1, 1, 4, 0, 0),
])
def test_stores(gpulib, cuda, M, N, K, pad, shift):
    import torch
    rng = np.random.default_rng(M + 3 * N + 7 * K + pad + shift)
    A, B = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((N, K)).astype(np.float32)
    dA, dB = torch.from_numpy(A).to(cuda), torch.from_numpy(B).to(cuda)
    ldc = N + pad
    buf = torch.full((shift + M * ldc + 8,), 7.0, device=cuda)
    err = torch.zeros(1, dtype=torch.int32, device=cuda)
    rc = gpulib.gpuisac_nn_gemm_bf16(M, N, K, ctypes.c_float(1.0), dA.data_ptr(), K, dB.data_ptr(), K, None, 0,
                                     buf.data_ptr() + 4 * shift, ldc, err.data_ptr(),
                                     torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    out = buf.cpu().numpy()
    got = out[shift:shift + M * ldc].reshape(M, ldc)
    want = bf16(A).astype(np.float64) @ bf16(B).astype(np.float64).T
    assert np.abs(got[:, :N] - want).max() <= 1e-4 * max(np.abs(want).max(), 1.0)
    assert (got[:, N:] == 7.0).all() and (out[:shift] == 7.0).all() and (out[shift + M * ldc:] == 7.0).all()
