"""Neighbour tables where the selection changes path (many equal distances,
too few threads for its bound, the most neighbours, each width of a thread's
share of the row) and at the edges of the distance tiles, against distances and
a stable sort in numpy: identical lists."""
import numpy as np
import pytest

from glphase_gb300 import model as mdl
from glphase_gb300.hmmlike import HMMLikeCUDA
from test_gpu_knn import gpu_knn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = HMMLikeCUDA(0)
    yield d
    d.cleanup()


def tract(a, b):
    """Common sites minus the longest run of agreement, per row of b."""
    S = b.shape[1]
    best = np.zeros(b.shape[0], np.int64)
    run = np.zeros(b.shape[0], np.int64)
    for m in range(S):
        run = np.where(b[:, m] == a[m], run + 1, 0)
        best = np.maximum(best, run)
    return S - best


def want(bits, K, samples, metric="hamming"):
    half = (K + 1) // 2
    out = []
    for s in samples:
        lists, taken = [], {2 * s, 2 * s + 1}
        for h in (2 * s, 2 * s + 1):
            d = ((bits != bits[h]).sum(axis=1) if metric == "hamming"
                 else tract(bits[h], bits))
            order = [int(i) for i in np.argsort(d, kind="stable") if int(i) not in taken]
            lists.append(order[:half])
            taken.update(lists[-1])
        out.append(np.stack(lists, axis=1).reshape(-1))
    return np.array(out, np.uint32)


def bits_of(H, S, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "same":
        return np.repeat(rng.integers(0, 2, size=(1, S)).astype(np.uint8), H, axis=0)
    if kind == "few":   # a handful of distinct haplotypes: ties by the hundred
        return rng.integers(0, 2, size=(7, S)).astype(np.uint8)[rng.integers(0, 7, size=H)]
    return (rng.random((H, S)) < rng.beta(0.5, 0.5, S)[None, :]).astype(np.uint8)


@pytest.mark.parametrize("H,S,K,kind", [
    (4, 1, 2, "random"), (6, 64, 3, "same"), (130, 65, 128, "random"), (254, 127, 20, "random"),
    (256, 128, 254, "few"), (258, 129, 31, "random"), (2400, 40, 100, "few"),
    (3000, 200, 200, "same"), (4096, 63, 2048, "random"), (4098, 193, 200, "random"),
    (8194, 90, 100, "random"), (20482, 130, 60, "random"), (20482, 33, 200, "few"),
])
def test_lists(dev, H, S, K, kind):
    bits = bits_of(H, S, kind, H + S)
    rng = np.random.default_rng(1)
    samples = sorted({0, H // 2 - 1, *rng.integers(0, H // 2, size=12).tolist()})
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, K)
    assert np.array_equal(got[samples], want(bits, K, samples))


@pytest.mark.parametrize("H,S,K,kind", [(130, 65, 40, "random"), (258, 31, 30, "few"),
                                        (258, 32, 30, "random"), (600, 33, 100, "random"),
                                        (5000, 200, 60, "random"), (70, 300, 20, "same")])
def test_tract_lists(dev, H, S, K, kind):
    bits = bits_of(H, S, kind, H + S)
    rng = np.random.default_rng(2)
    samples = sorted({0, H // 2 - 1, *rng.integers(0, H // 2, size=6).tolist()})
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, K, metric="tract")
    assert np.array_equal(got[samples], want(bits, K, samples, "tract"))


def test_common_sites_of_many_haplotypes(dev):
    """Frequency bounds at exact fractions of the haplotypes: a site counted one
    off changes the common set."""
    H, S, K = 3002, 150, 40
    rng = np.random.default_rng(3)
    bits = np.zeros((H, S), np.uint8)
    for m in range(S):
        bits[rng.permutation(H)[:10 * m], m] = 1
    lo, hi = 300 / H, 900 / H
    keep = (bits.sum(axis=0) >= 300) & (bits.sum(axis=0) <= 900)
    got = gpu_knn(dev, mdl.pack_haplotypes(bits), S, K, lo, hi)
    assert np.array_equal(got[[0, 700, 1500]], want(bits[:, keep], K, [0, 700, 1500]))


def want_words(words, K, samples):
    half = (K + 1) // 2
    out = []
    for s in samples:
        lists, taken = [], np.zeros(len(words), bool)
        taken[2 * s:2 * s + 2] = True
        for h in (2 * s, 2 * s + 1):
            d = np.bitwise_count(words ^ words[h]).sum(axis=1, dtype=np.int64)
            d[taken] = 1 << 20
            lists.append(np.argsort(d, kind="stable")[:half])
            taken[lists[-1]] = True
        out.append(np.stack(lists, axis=1).reshape(-1))
    return np.array(out, np.uint32)


@pytest.mark.parametrize("H,S,K", [(300, 65534, 40), (24002, 64, 100), (50000, 22000, 200)])
def test_words(dev, H, S, K):
    """The most sites (sums near 2^16), distances held a chunk at a time, and
    operand rows a slab at a time."""
    rng = np.random.default_rng(H)
    wn = (S + 63) // 64
    words = rng.integers(0, 2**64, size=(H, wn), dtype=np.uint64)
    words[:, -1] &= np.uint64((1 << (S - 64 * (wn - 1))) - 1 if S % 64 else 2**64 - 1)
    if H == 300:
        words[:100] = words[0]                     # equal haplotypes: a product of S
        words[100:200] = ~words[0]                 # and opposite ones: of -S
        words[100:200, -1] &= np.uint64((1 << (S - 64 * (wn - 1))) - 1)
        for i in range(200):                       # one to 200 sites apart
            words[i, :i // 64 + 1] ^= np.uint64((1 << (i % 64 + 1)) - 1)
    samples = [0, 1, 60, H // 4, H // 2 - 1]
    got = gpu_knn(dev, words, S, K)
    assert np.array_equal(got[samples], want_words(words, K, samples))
