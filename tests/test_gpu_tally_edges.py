"""Tallies and probabilities at the sizes where the kernels change path (rows of
whole vectors or not, rows that the registers hold or not, tiles of 64) and with
tallies whose sums wrap in 32 bits, against the oracle's restatement of
Impute::replace and numpy: identical."""
import numpy as np
import pytest

from glphase_gb300.hmmlike import HMMLikeCUDA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,S,offset", [
    (1, 1, 0), (3, 3, 0), (5, 4, 0), (5, 8, 1), (40, 63, 0), (33, 64, 0), (32, 65, 0),
    (3, 2048, 0), (2, 2052, 0), (2, 2049, 3), (2, 16384, 0), (2, 16388, 0), (2, 20001, 0),
])
def test_tally_and_result(oracle_lib, N, S, offset):
    import torch
    O = oracle_lib
    dev = HMMLikeCUDA(0)
    try:
        rng = np.random.default_rng(N * S + offset)
        wn = (S + 63) // 64
        cpu = rng.integers(0, 2**32, size=2 * N * S, dtype=np.uint64).astype(np.uint32)
        buf = torch.zeros(2 * N * S + offset, dtype=torch.int32, device="cuda")
        buf[offset:] = torch.from_numpy(cpu.view(np.int32)).cuda()
        ptr = buf.data_ptr() + 4 * offset
        for _ in range(3):
            haps = rng.integers(0, 2**64, size=(2 * N, wn), dtype=np.uint64)
            for s in range(N):
                O.lib().glpo_replace(haps.reshape(-1), wn, S, s, cpu)
            d = torch.from_numpy(haps.view(np.int64)).cuda()
            torch.cuda.synchronize()
            dev._c(dev.L.glp_tally(dev.ctx, d.data_ptr(), N, S, ptr))
            dev._c(dev.L.glp_finish(dev.ctx))
        assert np.array_equal(buf[offset:].cpu().numpy().view(np.uint32), cpu)
        prob = torch.full((S, 2 * N), -1.0, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        dev._c(dev.L.glp_result(dev.ctx, ptr, N, S, 3, prob.data_ptr()))
        dev._c(dev.L.glp_finish(dev.ctx))
        want = cpu.reshape(2 * N, S).T.astype(np.float32) * np.float32(1.0 / 3)
        assert np.array_equal(prob.cpu().numpy(), want)
    finally:
        dev.cleanup()
