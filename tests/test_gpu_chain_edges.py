"""The generation kernel where its chains' bookkeeping and the sites above the
last whole word can go wrong: cycle counts around the windows of draws (2 P
cycles of a chain, made P at a time), groups of a warp that leave it at different
times, every remainder of a word, and rescaling inside the remainder.

Decisions, quadruples and words against the oracle, and against the narrowest
speculation, exactly; log-likelihoods within 1e-5 of the oracle's (the
reference's binary32 arithmetic, impute.cpp:327-376, rounds a site's products
and sums about ten times, 6e-8 each; over S sites that grows as sqrt(S) against a
log-likelihood that grows as S).
"""
import numpy as np
import pytest

from glphase_gb300 import native as nat
from glphase_gb300.glpack import GLPack
from glphase_gb300.hmmlike import HMMLikeCUDA
from test_gpu_parity import REL_TOL, check_against_oracle, make_problem, run_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = HMMLikeCUDA(0)
    yield d
    d.cleanup()


def at_width(dev, lanes, *args, **kw):
    dev.set_lanes_per_sample(lanes)
    try:
        return run_gpu(dev, *args, **kw)
    finally:
        dev.set_lanes_per_sample(0)


@pytest.mark.parametrize("C", [0, 1, 2, 7, 8, 9, 31, 32, 33, 65, 130])
def test_windows_of_draws(dev, oracle_lib, C):
    m, haps, quad, props = make_problem(N=37, S=70, C=C, seed=C + 1)
    ref = at_width(dev, 1, m, haps, quad, props, 0.5, seed=9, gen=3)
    check_against_oracle(oracle_lib, m, haps, quad, props, 0.5, ref, 9, 3, check_work=False)
    for lanes in (2, 4, 8, 16, 32, 0):  # 0: teams of warps
        out = at_width(dev, lanes, m, haps, quad, props, 0.5, seed=9, gen=3)
        for key in ("quad", "acc", "hnew", "like"):
            assert np.array_equal(out[key], ref[key]), (lanes, key)
        assert np.array_equal(out["evals"], ref["evals"], equal_nan=True), lanes


@pytest.mark.parametrize("pen", [1e-9, 0.003, 0.02, 0.08, 0.25, 1.0])
def test_trees_of_every_shape(dev, oracle_lib, pen):
    """Penalties from chains that accept everything to ones that accept little, so
    that the wide groups' trees go from a line of acceptances over branched ones to
    a line of refusals, at cycle counts that end a round early; the rate that the
    kernel starts from is the generation before's."""
    for N, C in ((3, 100), (37, 47)):
        m, haps, quad, props = make_problem(N=N, S=130, C=C, seed=C)
        ref = at_width(dev, 1, m, haps, quad, props, pen, seed=4, gen=1)
        check_against_oracle(oracle_lib, m, haps, quad, props, pen, ref, 4, 1, check_work=False)
        for lanes in (16, 32, 0, 16, 32, 0):  # 0: teams of warps
            out = at_width(dev, lanes, m, haps, quad, props, pen, seed=4, gen=1)
            for key in ("quad", "acc", "hnew", "like"):
                assert np.array_equal(out[key], ref[key]), (lanes, key)
            assert np.array_equal(out["evals"], ref["evals"], equal_nan=True), lanes
            assert dev.counters()[2] == ref["acc"].sum()


@pytest.mark.parametrize("vq", [False, True])
@pytest.mark.parametrize("first", [0, 64, 192])
def test_every_remainder_of_a_word(dev, oracle_lib, first, vq):
    O = oracle_lib
    for left in [1, 2, 3, 4, 5, 7, 8, 9, 12, 31, 33, 40, 61, 62, 63]:
        S = first + left
        m, haps, quad, props = make_problem(N=9, S=S, C=9, seed=S)
        if not vq:
            out = run_gpu(dev, m, haps, quad, props, 1.0, seed=5, gen=2)
            check_against_oracle(O, m, haps, quad, props, 1.0, out, 5, 2, check_work=False)
            continue
        gp = GLPack(m.t, np.random.default_rng(left))
        packed, cb = gp.packed_gls(), gp.code_book()
        dev.copy_code_book_to_device(cb)
        dev.copy_packed_gls_to_device(packed)
        out = run_gpu(dev, m, haps, quad, props, 1.0, seed=5, flags=nat.GLP_GEN_VQ)
        pb = O.OracleProblem(haps, m.emit, m.t, m.tran, m.pc, 9, packed=packed, codebook=cb,
                             emit_mode=O.EMIT_VQ)
        tr = pb.trace(seed=5, generation=0)
        for s in range(m.N):
            like32, _, own, qf = O.replay_sample(pb, tr, s, quad, props, 1.0, out["acc"][s])
            rel = np.abs(out["evals"][s] - like32) / np.abs(like32)
            assert rel.max() <= REL_TOL, (S, s, rel.max())
            assert np.array_equal(qf, out["quad"][:, s])


@pytest.mark.parametrize("scale", [1e-3, 1e-8, 1e-12])
def test_rescaling_inside_the_remainder(dev, oracle_lib, scale):
    """Emissions that take the state below 2^-64 within a site, within four, and
    over several fours, in some samples and not in others."""
    m, haps, quad, props = make_problem(N=12, S=64 + 47, C=10, seed=21)
    m.emit = m.emit.copy()
    m.emit[::2, 70:100] *= np.float32(scale)
    m.emit[1::4, 101] *= np.float32(scale)
    pb = oracle_lib.OracleProblem(haps, m.emit, m.t, m.tran, m.pc, 10)
    tr = pb.trace(seed=6, generation=1)
    for lanes in (2, 8, 32):
        out = at_width(dev, lanes, m, haps, quad, props, 1.0, seed=6, gen=1)
        for s in range(m.N):
            like32, like64, _, qf = oracle_lib.replay_sample(pb, tr, s, quad, props, 1.0,
                                                             out["acc"][s])
            # at 1e-12 the binary32 reference leaves its own range for some quadruples
            # (0 times infinity: NaN); the binary64 one stands for it there
            ok = np.isfinite(like32)
            assert scale < 1e-8 or np.all(ok)
            assert np.all(np.isfinite(like64))
            for want, at in ((like64, slice(None)), (like32.astype(np.float64), ok)):
                rel = np.abs(out["evals"][s][at] - want[at]) / np.abs(want[at])
                assert rel.max() <= REL_TOL, (lanes, s, rel.max())
            assert np.array_equal(qf, out["quad"][:, s])


def test_uniforms_at_the_ends_of_their_range(dev):
    """The accept test takes the uniform rounded down to a float: traced uniforms
    that are 0, that lie between floats, that no float of the rule's range reaches,
    and next to 1, against the rule in binary64 (prop >= curr, or u < exp(d) for d =
    (prop - curr) pen above -37, or u = 0 below it), on either side of -37."""
    m, haps, quad, props = make_problem(N=16, S=150, C=24, seed=33)
    rng = np.random.default_rng(5)
    ends = np.array([0.0, 2.0**-53, 1e-300, 2.0**-40 + 2.0**-53, 0.5 - 2.0**-53, 0.5,
                     0.5 + 2.0**-53, 1 - 2.0**-53])
    u = ends[rng.integers(0, len(ends), (16, 24))]
    trace = (rng.integers(0, 4, (16, 24)).astype(np.uint8), u,
             rng.random((16, 150)).astype(np.float32))
    accepted = []
    for pen in (0.01, 1.0, 30.0):
        out = run_gpu(dev, m, haps, quad, props, pen, trace=trace)
        for s in range(16):
            curr = out["evals"][s, 0]
            for c in range(24):
                prop = out["evals"][s, c + 1]
                d = (prop - curr) * pen
                bound = 1.0 if d >= 0 else np.exp(d) if d > -37 or u[s, c] == 0 else 0.0
                if abs(bound - u[s, c]) > 3e-6 * bound:  # the exponential is binary32
                    assert out["acc"][s, c] == (d >= 0 or u[s, c] < bound), (pen, s, c)
                curr = prop if out["acc"][s, c] else curr
        accepted.append(out["acc"][u == 0.0].mean())
    assert accepted[0] == 1.0 and accepted[2] < 1.0


@pytest.mark.parametrize("lanes", [2, 8, 32])
def test_queue_of_uneven_chunks(dev, lanes):
    """More samples than the GPU holds groups (at 32 lanes), chunks not in the
    order of their sites: every sample is run once, in its own chunk."""
    import ctypes

    import torch
    from test_gpu_batch import Chunk
    chunks = [Chunk(dev, N, S, 3, seed=i + 1)
              for i, (N, S) in enumerate([(700, 40), (1101, 130), (3, 200), (997, 70)])]
    dev.set_lanes_per_sample(lanes)
    try:
        torch.cuda.synchronize()
        args = (nat.GenerationArgs * 4)(*[ch.args(0.5, 2) for ch in chunks])
        pbs = (ctypes.c_void_p * 4)(*[ch.pb for ch in chunks])
        dev._c(dev.L.glp_run_batch(dev.ctx, 4, pbs, args))
        dev._c(dev.L.glp_finish(dev.ctx))
        batched = [ch.outputs() for ch in chunks]
        for ch, out in zip(chunks, batched):
            ch.reset()
            dev.copy_tran_to_device(ch.m.tran)
            dev.copy_mutation_mat_to_device(ch.m.pc)
            dev.copy_emission_to_device(ch.m.emit, ch.m.t)
            torch.cuda.synchronize()
            a = ch.args(0.5, 2)
            dev._c(dev.L.glp_run_generation(dev.ctx, ctypes.byref(a)))
            dev._c(dev.L.glp_finish(dev.ctx))
            alone = ch.outputs()
            for k in ("quad", "like", "acc", "evals", "hnew"):
                assert np.array_equal(out[k], alone[k]), k
    finally:
        dev.set_lanes_per_sample(0)
        for ch in chunks:
            dev.L.glp_problem_destroy(ch.pb)
