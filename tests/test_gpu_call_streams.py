"""Calls on a stream of their own (non-blocking, as torch's side streams are):
tables, twiddles, texture handles and flags go through that stream.  A copy on
the legacy default stream would wait for what that one still runs (here a
kernel of a few hundred milliseconds), would not wait for what the caller's
stream still writes, and might arrive after the kernels that read it."""
import numpy as np
import pytest

from gpuisac import synth

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 1 << 30  # half a second at the SMs' highest clock


def _calls(cuda):
    """name -> a call on the current stream; every one is run with one geometry
    and then another, so that its tables are uploaded again"""
    import torch
    from gpuisac import align, averages, learned
    stacks = [synth.make_stack(60, D, 6, 2, 0.1, 0.4 * D, 5 + D) for D in (64, 72)]
    dev = [(torch.from_numpy(s.particles).to(cuda), torch.from_numpy(s.refs).to(cuda)) for s in stacks]
    rings = (25, 30)
    nets = [learned.ProposalNet(r, seed=3) for r in rings]
    embs = [learned.reference_embeddings(n, r, k) for n, (_, r), k in zip(nets, dev, rings)]
    groups = [(0, 25, 0, 3), (25, 35, 3, 3)]
    lists = torch.arange(3, dtype=torch.int32, device=cuda).repeat(60, 1).contiguous()
    peaks = torch.zeros(4, 60, 4, device=cuda)
    peaks[..., 0] = torch.linspace(0, 350, 60, device=cuda)
    bel = (torch.arange(60, device=cuda) % 4).int()

    def grouped(i):
        return align.multi_ref_align_groups_device(*dev[i], groups, rings[i], 2.0 - i, 2.0 - i)[:2]

    def proposals(i):
        return align.align_proposals_device(*dev[i], lists, rings[i], 2.0 - i, 2.0 - i)

    def search(i):
        r = learned.learned_align(*dev[i], nets[i], rings[i], 2.0 - i, 2.0 - i, k=3, ref_embed=embs[i])
        return r.ref, r.peak, r.params

    def average(i):
        return averages.class_averages_device(dev[i][0], peaks, bel, 0.3, 0.2)

    return {"groups": grouped, "proposals": proposals, "learned": search, "averages": average}


@pytest.mark.parametrize("name", ["groups", "proposals", "learned", "averages"])
def test_call_keeps_to_its_stream(gpulib, cuda, name):
    import torch
    call = _calls(cuda)[name]
    want = [[t.clone() for t in call(i)] for i in (0, 1)]  # (the work spaces have their sizes now)
    torch.cuda.synchronize()
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda._sleep(BUSY_CYCLES)  # the default stream is busy
    done.record()
    with torch.cuda.stream(side):
        got = [call(i) for i in (0, 1)]
        side.synchronize()
    waited = done.query()
    torch.cuda.synchronize()
    assert not waited, "the call waited for the default stream"
    for w, g in zip(want, got):
        for a, b in zip(w, g):
            assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())
