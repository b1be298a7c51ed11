"""hmm_work on the device against the oracle's restatement, every word of every
sample, at the sizes where its tiles, halves and blocks end: sites around
multiples of 8, 16, 64 and of a block's 32 samples, chunks of different lengths
in one batch, and sums outside the fast reciprocal's range.  Whole haplotype
words are compared, so one differently rounded product in ten million shows."""
import numpy as np
import pytest

import oracle as O
from glphase_gb300 import native as nat, synth
from glphase_gb300.hmmlike import HMMLikeCUDA

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def oracle_lib():
    O.build(ref=False)


def problem(N, S, seed, scale=None):
    w = synth.Workload("t", N=N, S=S, founders=6, depth=2.0, burnin=1, sampling=1, cycles=2,
                       seed=seed)
    m, haps = synth.initial_state(synth.generate(w))
    if scale is not None:
        m.emit = np.ascontiguousarray(m.emit * np.float32(scale)[None, :, None])
    return m, haps


def run(m, haps, pen, C=2, seed=5, generation=3):
    import ctypes as C_
    dev = HMMLikeCUDA(0)
    try:
        dev.copy_tran_to_device(m.tran)
        dev.copy_mutation_mat_to_device(m.pc)
        dev.copy_emission_to_device(m.emit, m.t)
        H = haps.shape[0]
        quad, props = synth.uniform_proposals(m.N, H, C, np.random.default_rng(seed))
        hnew, qo = haps.copy(), np.zeros_like(quad)
        a = nat.GenerationArgs()
        a.num_samples, a.num_sites, a.num_cycles, a.num_haps = m.N, m.S, C, H
        a.haps, a.hnew = haps.ctypes.data, hnew.ctypes.data
        a.hap_idxs_in, a.hap_idxs_out, a.props = (quad.ctypes.data, qo.ctypes.data,
                                                  props.ctypes.data)
        a.pen, a.seed, a.generation = pen, seed, generation
        dev._c(dev.L.glp_run_generation_host(dev.ctx, C_.byref(a)))
        return hnew, qo
    finally:
        dev.cleanup()


def check(m, haps, pen, samples=None):
    hnew, quad = run(m, haps, pen)
    for s in range(m.N) if samples is None else samples:
        u = O.work_uniforms(5, 3, s, m.S)
        ha, hb = O.hmm_work(m.emit[s], m.t[s], m.tran, m.pc, haps, quad[:, s], pen, u)
        assert np.array_equal(ha, hnew[2 * s]) and np.array_equal(hb, hnew[2 * s + 1]), s


@pytest.mark.parametrize("N", [1, 31, 32, 33, 65])
@pytest.mark.parametrize("S", [1, 7, 8, 9, 16, 17, 63, 64, 65, 200])
def test_edges(N, S):
    check(*problem(max(N, 2), S, 100 * N + S), 1.0)


@pytest.mark.parametrize("pen", [1.0, 0.140625])
def test_many_sites(pen):
    """4 million sites: enough that a contracted sum or a reciprocal one unit off
    changes a word."""
    check(*problem(1000, 4000, 9), pen)


@pytest.mark.parametrize("S", [40, 130])
def test_sums_outside_the_fast_reciprocal(S):
    """Emissions of 1e-39 (subnormal sums), 1e-45 (sums that round to zero or the
    smallest subnormal) and 1e38 at single sites of either half."""
    for site, f in ((3, 1e-39), (S - 2, 1e-39), (S // 2, 1e-45), (5, 1e38), (S - 5, 1e38)):
        scale = np.ones(S)
        scale[site] = f
        m, haps = problem(40, S, S, scale)
        check(m, haps, 1.0)
