"""Neighbour tables of panels whose rows fewer threads hold than a list has entries:
identical to distances and a stable sort in numpy on both sides of the rules that
choose the list's bound, and in times that grow with the lists' lengths and no faster.
Tract distances of few words, around the number up to which they are taken exactly."""
import time

import numpy as np
import pytest

from glphase_gb300 import model as mdl
from glphase_gb300.hmmlike import HMMLikeCUDA
from test_gpu_knn import gpu_knn
from test_gpu_knn_edges import bits_of, want
from test_gpu_knn_tract_forms import haplotypes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = HMMLikeCUDA(0)
    yield d
    d.cleanup()


@pytest.mark.parametrize("kind", ["random", "few", "same"])
@pytest.mark.parametrize("H,S,K", [(318, 90, 100), (320, 40, 316), (322, 40, 100), (322, 130, 320),
                                   (700, 64, 200), (1000, 300, 400), (1026, 33, 1024),
                                   (1400, 200, 1000), (2058, 70, 2048), (4094, 150, 1100),
                                   (4096, 150, 1100), (4098, 150, 1100)])
def test_lists(dev, H, S, K, kind):
    bits = bits_of(H, S, kind, H + K)
    rng = np.random.default_rng(K)
    samples = sorted({0, H // 2 - 1, *rng.integers(0, H // 2, size=8).tolist()})
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, K)
    assert np.array_equal(got[samples], want(bits, K, samples))


@pytest.mark.parametrize("kind", ["half", "tracts", "none"])
@pytest.mark.parametrize("S", [383, 384, 385, 448, 449, 512])
def test_tract_words(dev, S, kind):
    bits = haplotypes(1300, S, kind)
    samples = [0, 1, 325, 649]
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, 60, metric="tract")
    assert np.array_equal(got[samples], want(bits, 60, samples, "tract"))


def table_us(dev, H, S, K):
    import torch
    words = torch.from_numpy(mdl.pack_haplotypes(bits_of(H, S, "random", 7)).view(np.int64)).cuda()
    out = torch.zeros((H // 2, K), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(8):
        t = time.perf_counter()
        for _ in range(20):
            dev._c(dev.L.glp_knn_neighbors(dev.ctx, words.data_ptr(), H, S, K, 0.0, 1.0, 0,
                                           out.data_ptr()))
        dev._c(dev.L.glp_finish(dev.ctx))
        best = min(best, (time.perf_counter() - t) / 20 * 1e6)
    return best


@pytest.mark.parametrize("H,S,K", [(700, 64, 200), (1000, 1000, 400)])
def test_time(dev, H, S, K):
    dev._c(dev.L.glp_set_knn_metric(dev.ctx, 0))
    assert table_us(dev, H, S, K) < 1.7 * table_us(dev, H, S, 20)
