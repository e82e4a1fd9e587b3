"""Rounding of the class averages' sums.  Members at angle 0 and shift 0 are
their pixels themselves, so an average is the FP32 sum of known values: its
error against FP64 is no larger than that of runs of P / (4 resident CTAs)
members (8 to 256; two CTAs per SM at side 76) added one after another and the
runs added one after another, which numpy restates on the same values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_runs(v, run):
    """[n][...] float32 summed in runs of `run`, the runs' sums in order"""
    total = None
    for k in range(0, len(v), run):
        s = v[k].copy()
        for x in v[k + 1:k + run]:
            s = s + x
        total = s if total is None else total + s
    return total


@pytest.mark.parametrize("P,R", [(20000, 200), (10000, 100), (1000, 4), (300, 30), (2000, 200)])
def test_error_of_the_sums(gpulib, cuda, P, R):
    import torch
    from gpuisac.averages import class_averages_device
    D = 76
    g = torch.Generator(device=cuda).manual_seed(P)
    imgs = torch.randn(P, D, D, generator=g, device=cuda)
    bel = (torch.arange(P, device=cuda) % R).int()
    avg = class_averages_device(imgs, torch.zeros(R, P, 4, device=cuda), bel, 0.0, 0.2, False)[0].cpu().numpy()
    quarter_waves = 4 * 2 * torch.cuda.get_device_properties(cuda).multi_processor_count
    run = min(256, max(8, -(-P // quarter_waves)))
    ours, runs = [], []
    for r in range(0, R, max(1, R // 20)):
        v = imgs[r::R].cpu().numpy()
        exact = v.astype(np.float64).mean(0)
        ours.append(avg[r] - exact)
        runs.append(in_runs(v, run) * np.float32(1.0 / len(v)) - exact)
    rms = [float(np.sqrt(np.mean(np.square(e)))) for e in (ours, runs)]
    assert rms[0] <= rms[1], rms


def test_sums_that_overflow(gpulib, cuda):
    """An average whose sum leaves FP32's range is infinite, not NaN."""
    import torch
    from gpuisac.averages import class_averages_device
    imgs = torch.full((400, 20, 20), 3e38, device=cuda)
    imgs[200:] = -3e38
    bel = (torch.arange(400, device=cuda) // 100).int()
    avg = class_averages_device(imgs, torch.zeros(4, 400, 4, device=cuda), bel, 0.0, 0.2, False)[0]
    assert torch.isposinf(avg[:2]).all() and torch.isneginf(avg[2:]).all()
