"""The grouped FP32 products at the edges of their tiles: a training batch with
one particle, ragged counts, no particles, and products large
enough for the 64 x 64 tile, against the FP64 oracle.  Bounds: the network
tests' own (gradients 1e-4 of their largest entry, products 1e-5)."""
import ctypes

import numpy as np
import pytest

import nn_oracle as nno
from gpuisac import learned

pytestmark = pytest.mark.gpu


def _t(a, cuda, dtype=None):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype or torch.float32, device=cuda)


def _rel(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-30)


@pytest.mark.parametrize("B,R,rings,nk,hidden,emb", [(1, 2, 1, 4, 8, 4), (33, 65, 3, 11, 40, 36), (31, 5, 2, 16, 33, 17),
                                                     (600, 300, 35, 16, 256, 128)])
def test_training_batch(gpulib, cuda, B, R, rings, nk, hidden, emb):
    import torch
    net = learned.ProposalNet(rings, nk=nk, hidden=hidden, emb=emb, scale=7.0, seed=B, device=cuda)
    rng = np.random.Generator(np.random.PCG64(B + R))
    p = net.params()
    p["b1"] = 0.05 * rng.standard_normal(p["b1"].shape).astype(np.float32)
    p["b2"] = 0.05 * rng.standard_normal(p["b2"].shape).astype(np.float32)
    net.load_params(p)
    Xp = np.abs(rng.standard_normal((B, net.n_in))).astype(np.float32)
    Xr = np.abs(rng.standard_normal((R, net.n_in))).astype(np.float32)
    labels = rng.integers(0, R, B).astype(np.int32)
    net.grad.fill_(float("nan"))  # every entry is written
    loss = net.loss_and_grad(_t(Xp, cuda), _t(labels, cuda, torch.int32), _t(Xr, cuda))
    want_loss, want_g, _ = nno.loss_and_grads(p, Xp, Xr, labels, net.scale)
    assert abs(loss.cpu().numpy().mean() - want_loss) < 1e-5 * max(1.0, abs(want_loss))
    g = net.grads()
    for k in ("W1", "b1", "W2", "b2"):
        assert _rel(g[k], want_g[k]) < 1e-4, k


def test_no_particles_are_refused(gpulib, cuda):
    import torch

    from gpuisac import GpuIsacError
    net = learned.ProposalNet(2, nk=4, hidden=8, emb=4, seed=1, device=cuda)
    with pytest.raises(GpuIsacError):
        net.loss_and_grad(torch.empty((0, net.n_in), device=cuda), torch.empty(0, dtype=torch.int32, device=cuda),
                          torch.ones((3, net.n_in), device=cuda))


@pytest.mark.parametrize("M,N,K,ta,tb", [(1000, 700, 33, False, True), (700, 1000, 64, True, False), (960, 704, 1, False, False)])
def test_large_tile(gpulib, cuda, M, N, K, ta, tb):
    import torch
    rng = np.random.Generator(np.random.PCG64(M + N + K))
    A, B = rng.standard_normal((M, K)).astype(np.float32), rng.standard_normal((K, N)).astype(np.float32)
    dA, dB = _t(A.T if ta else A, cuda), _t(B.T if tb else B, cuda)
    C = torch.empty((M, N), device=cuda)
    rc = gpulib.gpuisac_nn_gemm(M, N, K, ctypes.c_float(1.0), dA.data_ptr(), *((1, M) if ta else (K, 1)), dB.data_ptr(),
                                *((1, K) if tb else (N, 1)), ctypes.c_float(0.0), C.data_ptr(), N,
                                torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    assert _rel(C.cpu().numpy(), A.astype(np.float64) @ B.astype(np.float64)) < 1e-5
