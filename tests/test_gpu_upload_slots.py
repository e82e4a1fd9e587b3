"""Host stacks on both sides of the size from which on an upload is staged in
larger slots (256 MiB), with pieces that do not end with an image, and a small
one after a large one: the drop-in call gives the bits of the call on device
tensors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(11_618,), (11_619,), (12_003, 700)])
def test_uploaded_stack_is_the_stack(gpulib, cuda, sizes):
    import torch
    from gpuisac import multi_ref_align
    from gpuisac.align import multi_ref_align_device
    D = 76  # 23,104 bytes an image: 256 MiB / 23,104 = 11,618.6
    rng = np.random.default_rng(sizes[0])
    for P in sizes:
        x, ref = rng.random((P, D, D), np.float32), rng.random((1, D, D), np.float32)
        pl, d = multi_ref_align(x, ref, 35, 0.0, 0.0)
        dd, pk = multi_ref_align_device(torch.from_numpy(x).to(cuda), torch.from_numpy(ref).to(cuda), 35, 0.0, 0.0)
        assert np.array_equal(d.reshape(1, P), dd.cpu().numpy())
        assert np.array_equal(pl.reshape(1, P, 4), pk.cpu().numpy())
