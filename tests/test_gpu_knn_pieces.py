"""Neighbour tables built in pieces: the library's host side compiled once more with
little memory to plan with gives the tables of the ordinary one, for chunks of
samples, slabs of operand rows on both sides, and both metrics."""
import ctypes as C
import glob
import os
import subprocess

import numpy as np
import pytest

from glphase_gb300 import build as B, native as nat

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(tmp_path_factory):
    """The library planning with at most 0 bytes: the least it can do with."""
    d = tmp_path_factory.mktemp("small")
    obj, so = str(d / "api.o"), str(d / "libsmall.so")
    subprocess.run([B.nvcc(), B.ARCH, *B.FLAGS, "-DGLP_KNN_LIMIT=0", "-c",
                    os.path.join(B.CSRC, "glp_api.cu"), "-o", obj], check=True)
    gens = sorted(glob.glob(os.path.join(B.OBJDIR, "glp_gen_*.o")))
    assert len(gens) == len(B.SOURCES) - 1
    subprocess.run([B.nvcc(), B.ARCH, "-shared", "-o", so, obj, *gens], check=True)
    return C.CDLL(so)


def table(L, words, S, K, metric):
    import torch
    H = len(words)
    ctx = C.c_void_p()
    assert L.glp_create(0, C.byref(ctx)) == 0
    try:
        haps = torch.from_numpy(words.view(np.int64)).cuda()
        out = torch.zeros((H // 2, 2 * ((K + 1) // 2)), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert L.glp_set_knn_metric(ctx, nat.KNN_METRICS[metric]) == 0
        for _ in range(2):
            assert L.glp_knn_neighbors(ctx, C.c_void_p(haps.data_ptr()), C.c_uint32(H),
                                       C.c_uint32(S), C.c_uint32(K), C.c_double(0.0),
                                       C.c_double(1.0), 0, C.c_void_p(out.data_ptr())) == 0
        assert L.glp_finish(ctx) == 0
        return out.cpu().numpy()
    finally:
        L.glp_destroy(ctx)


@pytest.mark.parametrize("metric", ["hamming", "tract"])
@pytest.mark.parametrize("H,S,K", [(60, 70, 20), (128, 64, 20), (130, 300, 40), (514, 200, 60),
                                   (1030, 1100, 100), (5000, 129, 200)])
def test_same_tables(small, H, S, K, metric):
    rng = np.random.default_rng(H + S)
    wn = (S + 63) // 64
    words = rng.integers(0, 2**64, size=(H, wn), dtype=np.uint64)
    words |= rng.integers(0, 2**64, size=(1, wn), dtype=np.uint64)
    if S % 64:
        words[:, -1] &= np.uint64((1 << (S % 64)) - 1)
    whole = table(nat.load(), words, S, K, metric)
    assert np.array_equal(table(small, words, S, K, metric), whole)
