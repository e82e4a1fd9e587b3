"""The spectra kernel at the ring counts where its pairing and its rounds of
16 FFT groups change (one ring, odd last rings, 16 and 17 pairs, the library's
largest count), sampled by the texture unit and by its emulation, against the
oracle (FP64).  The bound is the spectra tests': FP32 sampling and a
256-point FFT stay within 2e-5 of a ring's largest coefficient."""
import numpy as np
import pytest

from gpuisac import synth
from test_gpu_spectra import cfgs, check, decode, oracle_spectra, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("texture", ["1", "0"])
@pytest.mark.parametrize("D,NR", [(40, 1), (40, 2), (40, 3), (76, 31), (76, 33), (76, 34), (184, 88)])
def test_ring_counts(gpulib, cuda, oracle_mod, monkeypatch, D, NR, texture):
    monkeypatch.setenv("GPUISAC_TEXTURE", texture)
    st = synth.make_stack(2, D, 2, 0, 0.2, D * 0.4, 31 + NR)
    base = np.array([[0.375, -0.25], [-1.5, 0.8125]], np.float32)
    gcfg, ocfg = cfgs(2, 2, D, NR, 0.0)
    lay = oracle_mod.OrcLayout(2, gpulib.get_texture_limit(D), 2)
    sbj = decode(run_gpu(gpulib, cuda, st.particles, gcfg, False, base=base), False)
    check(sbj, oracle_spectra(oracle_mod, st.particles, ocfg, lay, False, base=base))
    ref = decode(run_gpu(gpulib, cuda, st.refs, gcfg, True), True)
    check(ref, oracle_spectra(oracle_mod, st.refs, ocfg, lay, True))
