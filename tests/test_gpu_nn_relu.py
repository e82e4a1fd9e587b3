"""gpuisac_nn_relu_backward: the gradient is kept where the activation is
positive and zero elsewhere (zero, negative, NaN), in place, one element more
and less than whole blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [0, 1, 255, 256, 257, 100_003])
def test_relu_backward(gpulib, cuda, n):
    import torch
    rng = np.random.default_rng(n)
    y, dy = rng.standard_normal(n + 1).astype(np.float32), rng.standard_normal(n + 1).astype(np.float32)
    y[::7] = 0.0
    y[3::11] = np.nan
    dev_y, dev_dy = torch.from_numpy(y).to(cuda), torch.from_numpy(dy).to(cuda)
    rc = gpulib.gpuisac_nn_relu_backward(dev_dy.data_ptr(), dev_y.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    want = dy.copy()
    want[:n][~(y[:n] > 0)] = 0.0
    assert np.array_equal(dev_dy.cpu().numpy(), want)  # (the element past the last untouched)
