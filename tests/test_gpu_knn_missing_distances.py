"""The neighbour lists when distances are missing: a wait of the product kernel
that runs out ends with false after its limit, and the selection behind it fills
the lists with "no haplotype" instead of reading what the distances' buffer holds;
rows with fewer entries than a list asks for leave the rest of it without
haplotypes, in both forms of the selection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SRC = r'''
#include "glp_knn_gemm.cuh"
__global__ void wait_kernel(unsigned long long limit, int *out) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    glp::mbar_init(&bar, 1);
    out[0] = glp::mbar_wait(&bar, 0, limit) ? 1 : 0;  // nothing arrives
  }
}
extern "C" int run_wait(unsigned long long limit, int *out) {
  wait_kernel<<<1, 32>>>(limit, out);
  return (int)cudaDeviceSynchronize();
}
extern "C" int run_select(const uint16_t *dist, uint32_t pitch, uint32_t H, uint32_t half,
                          uint32_t dmax, const int *error, uint32_t *nbr) {
  glp::knn_select_kernel<1><<<H / 2, glp::kKnnThreads>>>(dist, pitch, H, 0, half, dmax, error,
                                                         nbr);
  return (int)cudaDeviceSynchronize();
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from device_code import compile_launcher
    import ctypes as C
    L = compile_launcher(tmp_path_factory.mktemp("knn"), SRC)
    L.run_wait.argtypes = [C.c_ulonglong, C.c_void_p]
    L.run_select.argtypes = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_uint32,
                             C.c_void_p, C.c_void_p]
    return L


def select(lib, dist, half, dmax, flag):
    import torch
    H, pitch = dist.shape
    d = torch.from_numpy(dist.view(np.int16)).cuda()
    err = torch.tensor([flag], dtype=torch.int32, device="cuda")
    nbr = torch.zeros((H // 2, 2 * half), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_select(d.data_ptr(), pitch, H, half, dmax, err.data_ptr(),
                          nbr.data_ptr()) == 0
    return nbr.cpu().numpy().view(np.uint32)


def test_wait_that_nothing_ends(lib):
    import torch
    out = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert lib.run_wait(1_000_000, out.data_ptr()) == 0
    assert out.item() == 0


@pytest.mark.parametrize("half", [1, 50, 1000])
def test_lists_behind_a_failed_wait(lib, half):
    rng = np.random.default_rng(half)
    dist = rng.integers(0, 2**16, size=(2050, 2176)).astype(np.uint16)
    assert np.all(select(lib, dist, half, 64, flag=2) == 0xffffffff)
    assert np.all(select(lib, dist, half, 64, flag=3) == 0xffffffff)


@pytest.mark.parametrize("half", [2, 50, 1000])
@pytest.mark.parametrize("flag", [0, 1])  # 1: an index error of another launch
def test_rows_with_too_few_entries(lib, half, flag):
    """Three entries a row; the padding past the last haplotype holds distances."""
    H, pitch = 2050, 2176
    dist = np.full((H, pitch), 0xffff, np.uint16)
    dist[:, H:] = 1
    at = np.array([5, 900, 2049])
    dist[:, at] = [3, 1, 2]
    got = select(lib, dist, half, 64, flag)
    first, second = got[:, 0::2], got[:, 1::2]
    n = min(half, 3)
    assert np.all(first[:, :n] == np.array([900, 2049, 5])[:n])
    assert np.all(first[:, n:] >= H)
    if half == 2:  # one is left for the second list
        assert np.all(second[:, 0] == 5) and np.all(second[:, 1:] >= H)
    else:
        assert np.all(second >= H)
