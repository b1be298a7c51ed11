"""Teams of two and four warps a chain that take several samples in turn: launched
with fewer teams than samples, whatever width the host would pick, for emission rows
and codes, and normalisation every 8 and every 4 sites.  Evaluations, decisions,
quadruples and likelihoods equal to the narrowest speculation's, every sample once."""
import ctypes as C

import numpy as np
import pytest

from glphase_gb300 import native as nat
from glphase_gb300.glpack import GLPack
from glphase_gb300.hmmlike import HMMLikeCUDA
from test_gpu_parity import make_problem, run_gpu

pytestmark = pytest.mark.gpu

SRC = r'''
#include <string.h>
#include "glp_launch.h"
namespace glp {
template <class E, int kSub>
SingleFn team(int P) {
  return P == 64 ? generation_kernel<64, E, kSub> : generation_kernel<128, E, kSub>;
}
}
struct Launch {
  uint32_t N, S, C, H, vq, sub, P, blocks;
  const void *haps, *emit, *tran, *packed, *table, *quad_in, *props;
  void *quad_out, *like, *evals, *acc, *record;  // record: stats, counter, error
  double pen, rate;
  unsigned long long seed;
  unsigned generation;
};
extern "C" int run(const Launch *l) {
  glp::GenParams p;
  memset(&p, 0, sizeof(p));
  p.N = l->N; p.S = l->S; p.C = l->C; p.H = l->H; p.wn = (l->S + 63) / 64;
  p.haps = (const uint64_t *)l->haps;
  p.emit = (const float4 *)l->emit;
  p.tran4 = (const float4 *)l->tran;
  p.tranp = p.tran4 + (l->S + 1);
  p.packed = (const uint32_t *)l->packed;
  p.vq_table = (const float4 *)l->table;
  p.quad_in = (const uint32_t *)l->quad_in;
  p.quad_out = (uint32_t *)l->quad_out;
  p.props = (const uint32_t *)l->props;
  p.like_out = (double *)l->like;
  p.eval_trace = (double *)l->evals;
  p.accept_trace = (uint8_t *)l->acc;
  p.stats = (unsigned long long *)l->record;
  p.counter = (uint32_t *)(p.stats + glp::kStats);
  p.error = (int *)(p.counter + 1);
  p.samp_hi = l->H;
  p.pen = (float)l->pen;
  p.rate = (float)l->rate;
  p.seed = l->seed;
  p.generation = l->generation;
  const int P = (int)l->P;
  const glp::SingleFn fn =
      l->vq ? (l->sub == 4 ? glp::team<glp::EmitVQ, 2>(P) : glp::team<glp::EmitVQ, 1>(P))
            : (l->sub == 4 ? glp::team<glp::EmitF32, 2>(P) : glp::team<glp::EmitF32, 1>(P));
  const size_t smem = glp::stage_bytes(P);
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return -1;
  fn<<<l->blocks, glp::kThreads, smem>>>(p);
  if (cudaGetLastError() != cudaSuccess)
    return -2;
  return (int)cudaDeviceSynchronize();
}
'''


class Launch(C.Structure):
    _fields_ = ([(k, C.c_uint32) for k in ("N", "S", "C", "H", "vq", "sub", "P", "blocks")] +
                [(k, C.c_void_p) for k in ("haps", "emit", "tran", "packed", "table", "quad_in",
                                           "props", "quad_out", "like", "evals", "acc",
                                           "record")] +
                [("pen", C.c_double), ("rate", C.c_double), ("seed", C.c_ulonglong),
                 ("generation", C.c_uint)])


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from device_code import compile_launcher
    return compile_launcher(tmp_path_factory.mktemp("teams"), SRC)


@pytest.fixture(scope="module")
def dev():
    d = HMMLikeCUDA(0)
    yield d
    d.cleanup()


def tran_rows(tran):
    """The kernels' rows: (t0, t1, t2, t0 - t2), first and last the identity, then
    (t1, t2, t0 - t2, t0 - t2)."""
    S = len(tran)
    t = np.zeros((S + 1, 4), np.float32)
    t[1:S, :3] = tran[1:]
    t[1:S, 3] = tran[1:, 0] - tran[1:, 2]
    t[[0, S]] = [1, 0, 0, 1]
    return np.concatenate([t, t[:, [1, 2, 3, 3]]])


def code_table(codebook, pc):
    g0, g1 = codebook[:, 0].astype(np.float32), codebook[:, 1].astype(np.float32)
    g2 = np.maximum((np.float32(1) - g0) - g1, np.float32(0))
    return np.stack([((pc[i, 0] * g0 + pc[i, 1] * g1) + pc[i, 2] * g1) + pc[i, 3] * g2
                     for i in range(4)], axis=1).astype(np.float32)


def run_teams(lib, m, haps, quad, props, pen, P, blocks, sub, rate, vq=None):
    import torch
    N, S = m.N, m.S
    H, Cc = haps.shape[0], props.shape[0]

    def put(a):
        return torch.from_numpy(np.ascontiguousarray(a)).cuda()
    keep = dict(haps=put(haps.view(np.int64)), emit=put(m.emit.astype(np.float32)),
                tran=put(tran_rows(np.asarray(m.tran, np.float32))),
                quad_in=put(quad.astype(np.int32)), props=put(props.astype(np.int32)),
                quad_out=torch.full((4, N), -1, dtype=torch.int32, device="cuda"),
                like=torch.zeros(N, dtype=torch.float64, device="cuda"),
                evals=torch.full((N, Cc + 1), float("nan"), dtype=torch.float64, device="cuda"),
                acc=torch.zeros((N, max(Cc, 1)), dtype=torch.uint8, device="cuda"),
                record=torch.zeros(8, dtype=torch.int64, device="cuda"))
    if vq is not None:
        keep["packed"] = put(vq[0].view(np.int32))
        keep["table"] = put(code_table(vq[1], np.asarray(m.pc, np.float32)))
    torch.cuda.synchronize()
    a = Launch(N=N, S=S, C=Cc, H=H, vq=int(vq is not None), sub=sub, P=P, blocks=blocks, pen=pen,
               rate=rate, seed=9, generation=3)
    for k, t in keep.items():
        setattr(a, k, t.data_ptr())
    assert lib.run(C.byref(a)) == 0
    out = {k: keep[k].cpu().numpy() for k in ("like", "evals", "quad_out", "acc", "record")}
    assert out["record"].view(np.int32)[2 * 6 + 1] == 0  # no index error
    return out


@pytest.mark.parametrize("vq", [False, True])
@pytest.mark.parametrize("sub", [8, 4])
@pytest.mark.parametrize("P", [64, 128])
def test_several_samples_a_team(lib, dev, P, sub, vq):
    for N, S, Cc, blocks in ((37, 70, 47, 1), (37, 200, 9, 3), (8, 130, 130, 2), (5, 64, 0, 1)):
        m, haps, quad, props = make_problem(N=N, S=S, C=max(Cc, 1), seed=S)
        props = props[:Cc]
        gp, flags = None, 0
        if vq:
            pack = GLPack(m.t, np.random.default_rng(S))
            gp = (np.ascontiguousarray(pack.packed_gls(), np.uint32).reshape(-1),
                  np.asarray(pack.code_book(), np.float32).reshape(-1, 2))
            dev.copy_code_book_to_device(gp[1])
            dev.copy_packed_gls_to_device(gp[0])
            flags = nat.GLP_GEN_VQ
        dev.set_lanes_per_sample(1)
        dev.set_block_sites(sub)
        try:
            for pen, rate in ((1e-9, 0.9), (0.02, 0.5), (0.3, 0.12), (1.0, 0.0)):
                want = run_gpu(dev, m, haps, quad, props, pen, seed=9, gen=3, flags=flags)
                got = run_teams(lib, m, haps, quad, props, pen, P, blocks, sub, rate, gp)
                assert np.array_equal(got["quad_out"].view(np.uint32), want["quad"])
                assert np.array_equal(got["like"], want["like"])
                assert np.array_equal(got["evals"], want["evals"])
                assert np.array_equal(got["acc"][:, :Cc], want["acc"])
                assert got["record"][2] == want["acc"].sum()
        finally:
            dev.set_lanes_per_sample(0)
            dev.set_block_sites(0)
