"""GL codes where the device's binary32 filter has to hand over to the binary64
comparison (exact and near ties, repeated entries, points on entries, points
that are not numbers) and at the edges of the packing tiles, against the host
restatement: identical codes."""
import numpy as np
import pytest

from glphase_gb300 import glpack
from glphase_gb300.hmmlike import HMMLikeCUDA

pytestmark = pytest.mark.gpu


def pack(dev, gl, cb, bits):
    import torch
    N, S = gl.shape[:2]
    per = 32 // bits
    g = torch.from_numpy(gl).cuda()
    out = torch.zeros(((S + per - 1) // per, N), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    dev._c(dev.L.glp_vq_pack(dev.ctx, g.data_ptr(), N, S, cb.ctypes.data, cb.shape[0], bits,
                             out.data_ptr()))
    dev._c(dev.L.glp_finish(dev.ctx))
    w = out.cpu().numpy().view(np.uint32)
    codes = np.stack([(w >> np.uint32(32 - bits * (k + 1))) & np.uint32(2**bits - 1)
                      for k in range(per)], axis=1)       # [words][per][N]
    return codes.reshape(-1, N).T                          # [N][words * per]


@pytest.mark.parametrize("N,S,K,bits", [(1, 1, 16, 4), (32, 64, 16, 4), (33, 65, 16, 4),
                                        (31, 63, 5, 4), (65, 130, 4, 2), (40, 21, 16, 8)])
def test_codes_at_tile_edges(N, S, K, bits):
    dev = HMMLikeCUDA(0)
    try:
        rng = np.random.default_rng(N * S)
        gl = rng.dirichlet([0.4] * 3, size=(N, S)).astype(np.float32)
        cb = np.ascontiguousarray(rng.dirichlet([0.7] * 3, size=K)[:, :2].astype(np.float32))
        got = pack(dev, gl, cb, bits)
        rr, het = glpack._normalise(gl)
        assert np.array_equal(got[:, :S], glpack.nearest_code(cb, rr, het))
        first = glpack.nearest_code(cb, rr[:1, :1], het[:1, :1])[0, 0]
        assert np.all(got[:, S:] == first)                 # sites past the end
    finally:
        dev.cleanup()


def test_codes_of_ties():
    dev = HMMLikeCUDA(0)
    try:
        rng = np.random.default_rng(5)
        cb = np.zeros((16, 2), np.float32)
        cb[:4] = [(0, 1), (0, 0), (1, 0), (0, 0)]          # entry 3 repeats entry 1
        cb[4:8] = [(0.25, 0.25), (0.75, 0.25), (0.25, 0.75), (0.25, 0.25)]
        near = np.float32(0.5)
        cb[8:12] = [(near, 0.5), (np.nextafter(near, np.float32(1)), 0.5),
                    (near, np.nextafter(near, np.float32(1))), (near, 0.5)]
        cb[12:] = rng.random((4, 2), dtype=np.float32) * 0.5
        # points on entries, half-way between entries, one ulp off, and 0 / 0
        grid = np.array([(a, b) for a in (0, 0.125, 0.25, 0.375, 0.5, 0.75, 1)
                         for b in (0, 0.125, 0.25, 0.375, 0.5, 0.75, 1)], np.float32)
        pts = np.concatenate([grid, cb, np.nextafter(cb, np.float32(2)),
                              np.nextafter(cb, np.float32(-1)).clip(0)])
        gl = np.zeros((1, len(pts) + 1, 3), np.float32)
        gl[0, :-1, :2] = pts
        gl[0, :-1, 2] = 1 - pts.sum(axis=1, dtype=np.float32)
        gl = np.repeat(gl, 3, axis=0)                      # the last site is 0 / 0
        with np.errstate(invalid="ignore"):
            rr, het = glpack._normalise(gl)
        want = glpack.nearest_code(cb, rr, het)
        assert np.array_equal(pack(dev, gl, cb, 4)[:, :gl.shape[1]], want)
    finally:
        dev.cleanup()
