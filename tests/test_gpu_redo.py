"""Evaluations whose blocked pass may have lost range are made again site by site:
the same from emission rows and from codes of the same values, for lengths that end
on whole fours or not, close to the likelihoods of the shorter blocks that keep the
range, and at a bounded cost."""
import numpy as np
import pytest

from glphase_gb300 import model as mdl
from glphase_gb300.hmmlike import Engine
from test_gpu_team_queue import code_table

pytestmark = pytest.mark.gpu


def engine(N, S, vq, block, seed=5):
    """Confident genotypes that eight neighbouring sites of every haplotype
    contradict: with blocks of eight sites every evaluation leaves the range."""
    rng = np.random.default_rng(seed)
    H, wn = 2 * N, (S + 63) // 64
    mu = mdl.finish_mutation_rate(mdl.mutation_rate(H), H)
    pc = np.asarray(mdl.mutation_matrix(mu), np.float32)
    r = np.full(S, 2e-6)
    r[0] = 0.0
    tran = mdl.transition_from_distances(r)
    codebook = rng.dirichlet([4, 2, 1], size=16)[:, :2].astype(np.float32)
    codebook[0] = (1, 0)
    codes = rng.integers(1, 16, size=(N, S)).astype(np.uint32)
    codes[:, 128:136] = 0
    bits = (rng.random((H, S)) < 0.3).astype(np.uint8)
    bits[:, 128:136] = 1
    packed = np.zeros(((S + 7) // 8, N), np.uint32)
    for m in range(S):
        packed[m // 8] |= codes[:, m] << np.uint32(28 - 4 * (m % 8))
    emit = code_table(codebook, pc)[codes]
    prob = np.zeros((N, S, 3), np.float32)
    prob[..., :2] = codebook[codes]
    prob[..., 2] = np.maximum((1 - prob[..., 0]) - prob[..., 1], 0)
    return Engine(emit, prob, tran, pc, mdl.pack_haplotypes(bits), 60, lanes=8,
                  packed=packed.reshape(-1) if vq else None, codebook=codebook if vq else None,
                  block_sites=block)


def run(eng, g, work=False):
    eng.launch(eng.args(None, None, 1.0, 3, g, work=work))
    eng.finish()
    return eng.like.cpu().numpy(), eng.quad.cpu().numpy()


@pytest.mark.parametrize("S", [193, 255, 256, 1001, 1003])
def test_rows_and_codes(S):
    out = [run(engine(40, S, vq, 8), 2) for vq in (False, True)]
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    eng = engine(40, S, False, 8)
    run(eng, 2)
    ev, redo = (eng.dev.counters()[i] for i in (0, 3))
    assert redo >= ev > 0  # lanes past a chain's end too
    four = engine(40, S, False, 4)
    like, quad = run(four, 2)
    assert four.dev.counters()[3] == 0
    same = (quad == out[0][1]).all(axis=0)  # a near tie may go the other way
    assert same.mean() > 0.9
    np.testing.assert_allclose(like[same], out[0][0][same], rtol=1e-6)


@pytest.mark.parametrize("vq", [False, True])
def test_time(vq):
    ms = {}
    for block in (8, 4):
        eng = engine(400, 2048, vq, block)
        for g in range(4):
            run(eng, 2)
        ms[block] = min(eng.dev.kernel_times(4)[0])
    # every evaluation made again: 5.7 and 5.3 times as long, 8.1 and 8.9 with a site at a time
    assert ms[8] < 7.0 * ms[4]
