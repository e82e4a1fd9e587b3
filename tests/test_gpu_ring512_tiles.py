"""The 512-sample contraction at the edges of its tiles (4, 8 and 16 references
per CTA; row and reference counts that leave tiles part empty; ring counts
around the 4 rings of a stage) against the FP64 oracle, and its reference
blocks (work space for fewer references than the call has) against one block."""
import numpy as np
import pytest

from gpuisac import synth

from test_gpu_align import compare
from test_gpu_ring512 import oracle_512

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,NR,rng", [(1, 1, 1, 0.0), (9, 4, 4, 1.0), (5, 5, 5, 1.0), (7, 8, 13, 1.0), (2, 9, 3, 2.0),
                                        (7, 17, 8, 1.0), (3, 33, 9, 0.0)])
def test_tiles_match_oracle(gpulib, cuda, oracle_mod, P, R, NR, rng):
    from gpuisac import multi_ref_align
    D = 40
    st = synth.make_stack(P, D, R, int(rng), 0.2, D * 0.4, 900 + P + R)
    pl, d = multi_ref_align(st.particles, st.refs, NR, rng, rng, ring_len=512)
    peak_o, d_o = oracle_512(oracle_mod, st.particles, st.refs, NR, rng, gpulib.get_texture_limit(D))
    compare(pl.reshape(R, P, 4), d, peak_o, d_o, ring_num=NR, ring_len=512)


def test_reference_blocks_equal_one_block(gpulib, cuda):
    from gpuisac import multi_ref_align
    st = synth.make_stack(3, 40, 90, 3, 0.2, 16.0, 41)
    pl, d = multi_ref_align(st.particles, st.refs, 9, 3.0, 3.0, ring_len=512)
    # a share of free memory that holds about 70 references' ring sums of one particle
    pl2, d2 = multi_ref_align(st.particles, st.refs, 9, 3.0, 3.0, ring_len=512, mem_request=1e-4)
    assert np.array_equal(d, d2) and np.array_equal(pl, pl2)
