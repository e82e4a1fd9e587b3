"""CCF tile shapes as they are asked for: the autotuner times every candidate
itself also on a sample of few work items, a choice of 4 contraction warps is
kept where items hold one particle, and every shape gives the general kernel's
bits."""
import numpy as np
import pytest

from gpuisac import synth
from gpuisac.align import (align_proposals_device, autotune_ccf, ccf_launched_name, multi_ref_align_device)

pytestmark = pytest.mark.gpu


def device_stack(cuda, P, D, R, shift, seed):
    import torch
    st = synth.make_stack(P, D, R, shift, 0.1, 0.4 * D, seed=seed)
    return torch.from_numpy(st.particles).to(cuda), torch.from_numpy(st.refs).to(cuda)


@pytest.mark.parametrize("P,R,NR,variants", [(128, 12, 27, ("ws8", "ws4", "tmem")), (40, 3, 45, ("ws8", "ws4"))])
def test_autotuner_runs_what_it_names(gpulib, cuda, P, R, NR, variants):
    """(128 x 12: 384 particle tiles, fewer than SMs x 4; 36 rings and more have no single-phase kernel)"""
    parts, refs = device_stack(cuda, P, 2 * NR + 8, R, 1, 5)
    rep = autotune_ccf(parts, refs, NR, 1.0, 1.0, n_sample=P)
    names = [e.rsplit(" ", 2)[0] for e in rep.split("; ") if not e.startswith("chosen")]
    assert sorted(names) == sorted(f"{v}/ppc{n}" for v in variants for n in (4, 8, 16))


@pytest.mark.parametrize("NR", [28, 44])
@pytest.mark.parametrize("warps", ["4", "8"])
def test_warps_are_kept_for_one_particle_items(gpulib, cuda, monkeypatch, NR, warps):
    import torch
    parts, refs = device_stack(cuda, 50, 2 * NR + 8, 9, 2, 6)
    lists = torch.from_numpy(np.stack([np.roll(np.arange(9), i)[:7] for i in range(50)]).astype(np.int32)).to(cuda)

    def run():
        full = multi_ref_align_device(parts, refs, NR, 2.0, 2.0, contraction_mode="fp32")
        name = ccf_launched_name()
        some = align_proposals_device(parts, refs, lists, NR, 2.0, 2.0)
        return (name, ccf_launched_name()), [t.cpu().numpy() for t in (*full, *some)]

    monkeypatch.setenv("GPUISAC_CCF_KERNEL", "general")
    (a, b), want = run()
    assert a.startswith("general/") and b.startswith("general/")
    monkeypatch.setenv("GPUISAC_CCF_KERNEL", "ws")
    monkeypatch.setenv("GPUISAC_CCF_WS_WARPS", warps)
    names, got = run()
    assert names == (f"ws{warps}/ppc1", f"ws{warps}/ppc1")
    for w, g in zip(want, got):
        assert np.array_equal(w, g)
