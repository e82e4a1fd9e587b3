"""Products with a short K (csrc/nn.cu) at the edges of the rule that gives them
their own kernel: K of 16 / 17, 24 / 25, 32 / 33, 48 / 49, 32 / 33 columns, one tile
fewer than SMs, ragged rows and columns, every pair of layouts, beta.  Within
the FP32 bound of a sum of K products in order, (K + 3) 2^-24 sum |a b|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (8, 8, 0), (65, 70, 16), (65, 70, 17), (9700, 8, 16), (9728, 64, 17), (9600, 64, 24),
                                   (9729, 65, 24), (9729, 65, 25), (9729, 65, 32), (9729, 65, 33), (9729, 33, 32), (9729, 32, 32), (20001, 32, 48), (20001, 33, 48), (20001, 32, 49), (70000, 3, 5)])
@pytest.mark.parametrize("ta,tb,beta", [(False, True, 0.0), (True, False, 0.0), (False, False, 2.0), (True, True, -1.0)])
def test_short_products(gpulib, cuda, M, N, K, ta, tb, beta):
    import torch
    g = torch.Generator(device=cuda).manual_seed(M + N + K)

    def rnd(*s):
        return torch.randn(*s, generator=g, device=cuda)

    A, B, C = rnd(*((max(K, 1), M) if ta else (M, max(K, 1)))), rnd(*((N, max(K, 1)) if tb else (max(K, 1), N))), rnd(M, N)
    a, b = (A.t() if ta else A)[:, :K].double(), (B.t() if tb else B)[:K].double()
    want = 0.5 * (a @ b) + beta * C.double()
    bound = (K + 3) * 2.0**-24 * (0.5 * (a.abs() @ b.abs()) + abs(beta) * C.double().abs()) + 1e-30
    rc = gpulib.gpuisac_nn_gemm(M, N, K, ctypes.c_float(0.5), A.data_ptr(), *((1, M) if ta else (max(K, 1), 1)),
                                B.data_ptr(), *((1, max(K, 1)) if tb else (N, 1)), ctypes.c_float(beta), C.data_ptr(), N,
                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert bool(((C.double() - want).abs() <= bound).all())
