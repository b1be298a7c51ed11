"""Sums outside the fast reciprocal's range cost hmm_work the steps around them, not
the whole block: the haplotypes are the oracle's where the sums leave the range for
a site and come back (2^-126 to 2^-128, 2^126 and above), at every place of a tile, and
the time stays below twice that of ordinary emissions (a block that started over,
one warp with both recursions in turn, took ten times as long), also where the state
is not finite from a site on, as the reference's is after a sum below 2^-128."""
import numpy as np
import pytest

from glphase_gb300 import hmmlike, synth
from test_gpu_work_exact import check, oracle_lib, problem  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [21, 150])
@pytest.mark.parametrize("factor", [2.0**-127, 2.0**127])
def test_sums_that_come_back(S, factor):
    for site in list(range(0, 18)) + [S - 1, S - 2, S - 9]:
        scale = np.ones(S)
        scale[site] = factor
        if site % 3 == 0 and site + 5 < S:
            scale[site + 5] = 1 / factor
        check(*problem(33, S, S + site, scale), 1.0, samples=(0, 7, 31, 32))


@pytest.mark.parametrize("N,S", [(40, 1024), (3000, 1024)])
@pytest.mark.parametrize("factor", [2.0**-127, 1e-39])
def test_time(N, S, factor):
    w = synth.Workload("t", N=N, S=S, founders=6, depth=2.0, burnin=1, sampling=1, cycles=2,
                       seed=N)
    m, haps = synth.initial_state(synth.generate(w))
    best = []
    for f in (1.0, factor):
        emit = m.emit.copy()
        emit[:, S // 3] *= np.float32(f)
        eng = hmmlike.Engine(emit, m.t, m.tran, m.pc, haps, 2)
        try:
            for g in range(8):
                eng.launch(eng.args(None, None, 1.0, 1, g))
                eng.finish()
            best.append(min(eng.dev.kernel_times(5)[1]))
        finally:
            eng.dev.cleanup()
    assert best[1] < 2 * best[0], best
