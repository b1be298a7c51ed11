"""The allocation-free entry point picks its speculation width for what its rows
cost, as the context's entry point does: without hmm_work its scratch bounds no
emission rows, and rows beyond L2 want wider groups.  The width changes no result,
so it shows in the time: both entry points run the same generation, and the
allocation-free one may take at most 1.15 times as long (it has one short launch
more; 4 lanes in place of 8 take 1.35 to 1.7 times as long here)."""
import ctypes as C
import time

import numpy as np
import pytest

from glphase_gb300 import native as nat, synth, synth_device
from glphase_gb300.hmmlike import HMMLikeCUDA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,S", [(20000, 512), (15000, 2048)])
def test_rows_beyond_l2(N, S):
    import torch
    w = synth.Workload("width", N=N, S=S, founders=40, depth=4.0, burnin=8, sampling=16)
    ch = synth_device.generate(w, N, S, 3)
    tran = torch.from_numpy(np.ascontiguousarray(ch.tran)).cuda()
    pc = np.ascontiguousarray(ch.pc, dtype=np.float32)
    quad = torch.zeros((4, N), dtype=torch.int32, device="cuda")
    like = [torch.zeros(N, dtype=torch.float64, device="cuda") for _ in range(2)]
    dev = HMMLikeCUDA(0)
    try:
        dev.copy_tran_to_device(np.ascontiguousarray(ch.tran, dtype=np.float32))
        dev.copy_mutation_mat_to_device(pc)
        dev.copy_emission_to_device(ch.emit.cpu().numpy(), ch.prob.cpu().numpy())
        torch.cuda.synchronize()

        def args(out):
            a = nat.GenerationArgs()
            a.num_samples, a.num_sites, a.num_cycles, a.num_haps = N, S, 100, ch.H
            a.haps, a.hap_idxs_out = ch.haps.data_ptr(), quad.data_ptr()
            a.like_out = out.data_ptr()
            a.pen, a.seed, a.generation, a.flags = 1.0, 1, 5, nat.GLP_GEN_NO_WORK
            return a

        def own():
            a = args(like[0])
            dev._c(dev.L.glp_run_generation(dev.ctx, C.byref(a)))
            dev._c(dev.L.glp_finish(dev.ctx))

        def noalloc():
            a = args(like[1])
            assert dev.L.glp_run_generation_noalloc(C.byref(a), tran.data_ptr(), pc.ctypes.data,
                                                    ch.emit.data_ptr(), None, None) == nat.GLP_OK

        best = {}
        for f in (own, noalloc):
            times = []
            for _ in range(8):
                t = time.perf_counter()
                f()
                times.append(time.perf_counter() - t)
            best[f] = min(times[2:])
        assert torch.equal(like[0], like[1])
        assert best[noalloc] <= 1.15 * best[own], (best[noalloc], best[own])
    finally:
        dev.cleanup()
