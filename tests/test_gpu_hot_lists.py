"""Neighbour lists over a few sites hold the same few haplotypes for all samples (equal
distances go to the lowest index), so that all warps read the same lines of the panel:
a generation from them takes no longer than one with proposals from everywhere."""
import numpy as np
import pytest

from glphase_gb300 import synth, synth_device
from glphase_gb300.hmmlike import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,S,K", [(584, 9, 70), (256, 9, 70)])
def test_time(N, S, K):
    import torch
    w = synth.Workload("hot", N=N, S=S, founders=21, depth=4.0, burnin=8, sampling=16)
    ch = synth_device.generate(w, N, S, 5)
    torch.cuda.synchronize()
    ms = {}
    for k in (0, K):
        eng = Engine(ch.emit.cpu().numpy(), ch.prob.cpu().numpy(), ch.tran, ch.pc,
                     ch.haps.cpu().numpy().view(np.uint64), 100)
        nbr = eng.knn(k) if k else None
        for g in range(14):
            eng.launch(eng.args(None, None, 1.0, 5, g, neighbors=nbr))
            eng.swap()
            eng.finish()
        ms[k] = min(eng.dev.kernel_times(10)[0])
    assert ms[K] < 1.25 * ms[0]
