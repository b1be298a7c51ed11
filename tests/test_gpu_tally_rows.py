"""Tallies of rows of any length and alignment (vectors of each row's own, single
sites at its ends, one to four vectors a thread, rows read twice), and probabilities
around the size from which tiles are turned: as the oracle and numpy give them.  Rows
that are short, or no multiple of four sites, take about as long as their neighbours
that are neither."""
import numpy as np
import pytest

from glphase_gb300.hmmlike import HMMLikeCUDA

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    import torch
    d = HMMLikeCUDA(0)
    st = torch.cuda.Stream()
    d._c(d.L.glp_set_stream(d.ctx, st.cuda_stream))
    d.torch_stream = st
    yield d
    d.cleanup()


def tally(dev, haps, N, S, ptr):
    dev._c(dev.L.glp_tally(dev.ctx, haps.data_ptr(), N, S, ptr))


def result(dev, ptr, N, S, prob):
    dev._c(dev.L.glp_result(dev.ctx, ptr, N, S, 3, prob.data_ptr()))


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 6, 7, 11, 61, 63, 66, 67, 125, 127, 129, 130, 255,
                               258, 509, 511, 513, 515, 518, 1023, 1025, 1027, 2049, 4099, 16383,
                               16387, 16390, 20003])
def test_rows(oracle_lib, dev, S, offset):
    import torch
    N, wn = 3, (S + 63) // 64
    rng = np.random.default_rng(4 * S + offset)
    cpu = rng.integers(0, 2**32, size=2 * N * S, dtype=np.uint64).astype(np.uint32)
    buf = torch.full((2 * N * S + offset + 8,), 77, dtype=torch.int32, device="cuda")
    buf[offset:offset + 2 * N * S] = torch.from_numpy(cpu.view(np.int32)).cuda()
    for _ in range(2):
        haps = rng.integers(0, 2**64, size=(2 * N, wn), dtype=np.uint64)
        for s in range(N):
            oracle_lib.lib().glpo_replace(haps.reshape(-1), wn, S, s, cpu)
        d = torch.from_numpy(haps.view(np.int64)).cuda()
        torch.cuda.synchronize()
        tally(dev, d, N, S, buf.data_ptr() + 4 * offset)
        dev._c(dev.L.glp_finish(dev.ctx))
    got = buf.cpu().numpy()
    assert np.array_equal(got[offset:offset + 2 * N * S].view(np.uint32), cpu)
    assert (got[:offset] == 77).all() and (got[offset + 2 * N * S:] == 77).all()


@pytest.mark.parametrize("N,S", [(512, 255), (512, 256), (512, 257), (1, 131072), (1, 131073),
                                 (131072, 1), (131073, 1), (2100, 63), (2100, 64), (2100, 65),
                                 (33, 4001), (64, 6400)])
def test_result(dev, N, S):
    import torch
    rng = np.random.default_rng(N + S)
    cpu = rng.integers(0, 2**32, size=(2 * N, S), dtype=np.uint64).astype(np.uint32)
    hsum = torch.from_numpy(cpu.view(np.int32)).cuda()
    prob = torch.full((S + 1, 2 * N), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    result(dev, hsum.data_ptr(), N, S, prob)
    dev._c(dev.L.glp_finish(dev.ctx))
    got = prob.cpu().numpy()
    assert np.array_equal(got[:S], cpu.T.astype(np.float32) * np.float32(1.0 / 3))
    assert (got[S] == -1.0).all()


def time_us(dev, what, N, S, n=50):
    import torch
    haps = torch.randint(-2**62, 2**62, (2 * N, (S + 63) // 64), device="cuda")
    hsum = torch.randint(0, 20, (2 * N, S), device="cuda", dtype=torch.int32)
    prob = torch.zeros((S, 2 * N), device="cuda")
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(8):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record(dev.torch_stream)
        for _ in range(n):
            if what == "tally":
                tally(dev, haps, N, S, hsum.data_ptr())
            else:
                result(dev, hsum.data_ptr(), N, S, prob)
        b.record(dev.torch_stream)
        b.synchronize()
        best = min(best, a.elapsed_time(b) / n * 1e3)
    return best


@pytest.mark.parametrize("N,S,even", [(8000, 101, 100), (20000, 3, 64), (4000, 4097, 4096)])
def test_tally_time(dev, N, S, even):
    assert time_us(dev, "tally", N, S) < 1.6 * time_us(dev, "tally", N, even)


def test_result_time(dev):
    # few entries in less time than the least number that is turned in tiles
    assert time_us(dev, "result", 500, 3) < 0.9 * time_us(dev, "result", 1100, 120)
