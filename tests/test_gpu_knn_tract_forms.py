"""Tract-length neighbour tables over haplotypes with short runs, long ones and
hardly any, at the words, tiles and distances where the kernel changes its form:
the first eight words, few tiles or many, and distances held a chunk of samples at
a time (more than 23,000 haplotypes).  Identical lists to numpy's."""
import numpy as np
import pytest

from glphase_gb300 import model as mdl
from glphase_gb300.hmmlike import HMMLikeCUDA
from test_gpu_knn import gpu_knn
from test_gpu_knn_edges import want

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = HMMLikeCUDA(0)
    yield d
    d.cleanup()


def haplotypes(H, S, kind):
    rng = np.random.default_rng(H + S)
    if kind == "half":      # agree at half of the sites
        return rng.integers(0, 2, (H, S)).astype(np.uint8)
    if kind == "tracts":    # mosaics with a few errors
        src = rng.integers(0, 6, (H, S // 50 + 1)).repeat(50, axis=1)[:, :S]
        out = rng.integers(0, 2, (6, S)).astype(np.uint8)[src, np.arange(S)[None, :]]
        return out ^ (rng.random((H, S)) < 0.02)
    # every other site differs between half of the pairs: longest runs of 0 and 1
    rows = np.stack([np.zeros(S), np.ones(S), np.arange(S) % 2, 1 - np.arange(S) % 2])
    return rows[rng.integers(0, 4, H)].astype(np.uint8)


@pytest.mark.parametrize("kind", ["half", "tracts", "none"])
@pytest.mark.parametrize("H,S", [(130, 3), (130, 500), (130, 512), (130, 513), (130, 576),
                                 (130, 1100), (700, 640), (900, 640), (1300, 512), (1300, 577),
                                 (1300, 1090), (24002, 70), (24002, 600)])
def test_lists(dev, H, S, kind):
    bits = haplotypes(H, S, kind)
    samples = [0, 1, H // 4, H // 2 - 1]
    if H > 24000:  # the last samples of a chunk and the first of the next
        samples += [2784, 2785, 2786, 2787, 2788, 2789, 2790]
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, 60, metric="tract")
    assert np.array_equal(got[samples], want(bits, 60, samples, "tract"))
