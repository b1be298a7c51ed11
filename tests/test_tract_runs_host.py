"""The open-run form of the kNN tract-length logic (glp_tract.h: tract_extend32
and tract_inside32 for words whose sites are all common, tract_extend for the
others, as knn_tract_dist_kernel runs them) compiled for the host and checked against the
oracle's Haplotype::MaxTractLen restatement: run lengths around every threshold
of the 32-bit form (7, 8, 14 to 17, 30 to 33) inside words and across them, and random
words."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include "glp_tract.h"
extern "C" uint32_t run_dist(const uint64_t *a, const uint64_t *b, const uint64_t *m, uint32_t wn) {
  glp::OpenRun r{0, glp::kRunFloor};
  glp::Tract t{0, 0, 0, 0};
  uint32_t common = 0;
  for (uint32_t w = 0; w < wn; ++w) {
    common += glp::tract_popc(m[w]);
    if (m[w] == ~0ull) {
      glp::tract_extend32(r, (uint32_t)(a[w] ^ b[w]));
      glp::tract_extend32(r, (uint32_t)((a[w] ^ b[w]) >> 32));
    } else {
      glp::tract_extend(r, (a[w] ^ b[w]) & m[w], m[w]);
    }
  }
  for (uint32_t w = 0; w < wn; ++w)
    if (m[w] == ~0ull) {
      glp::tract_inside32(r.best, (uint32_t)(a[w] ^ b[w]));
      glp::tract_inside32(r.best, (uint32_t)((a[w] ^ b[w]) >> 32));
    }
  for (uint32_t w = 0; w < wn; ++w)
    t = glp::tract_join(t, glp::tract_word((a[w] ^ b[w]) & m[w], m[w]));
  return common - (r.best == glp::kRunFloor ? t.best : r.best);
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("runs")
    src, so = d / "runs.cpp", d / "libruns.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wno-unknown-pragmas", "-I",
                    os.path.join(ROOT, "glphase_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = C.CDLL(str(so))
    p = np.ctypeslib.ndpointer(dtype=np.uint64, flags="C_CONTIGUOUS")
    L.run_dist.restype = C.c_uint32
    L.run_dist.argtypes = [p, p, p, C.c_uint32]
    return L


def pack(bits):
    by = np.packbits(bits.reshape(-1, 8), axis=1, bitorder="little").reshape(-1)
    return by.view("<u8").astype(np.uint64)


def test_runs_at_every_threshold(lib, oracle_lib):
    rng = np.random.default_rng(4)
    full = np.full(4, 2**64 - 1, np.uint64)
    a = np.zeros(4, np.uint64)
    for length in (1, 2, 6, 7, 8, 9, 13, 14, 15, 16, 17, 29, 30, 31, 32, 33, 47, 63, 64, 65, 100):
        for start in range(0, 256 - length, 3):
            x = np.ones(256, np.uint8)          # disagreements but for runs
            x[start:start + length] = 0
            for _ in range(3):                  # and shorter ones before and after
                s, n = int(rng.integers(0, 250)), int(rng.integers(0, 18))
                keep = x.copy()
                keep[s:s + n] = 0
                x = keep if rng.random() < 0.7 else x
            b = pack(x)
            assert lib.run_dist(a, b, full, 4) == 256 - oracle_lib.max_tract(a, b, full)


def test_random_words(lib, oracle_lib):
    rng = np.random.default_rng(5)
    for t in range(3000):
        wn = int(rng.integers(1, 9))
        a = rng.integers(0, 2**64, wn, dtype=np.uint64)
        b = a ^ pack((rng.random(64 * wn) < rng.choice([0.02, 0.1, 0.25, 0.5])).astype(np.uint8))
        m = np.full(wn, 2**64 - 1, np.uint64)
        if t % 3 == 1:
            m = pack((rng.random(64 * wn) < 0.7).astype(np.uint8))
        elif t % 3 == 2:
            m[-1] = np.uint64((1 << int(rng.integers(1, 64))) - 1)
        common = sum(bin(int(x)).count("1") for x in m)
        assert lib.run_dist(a, b, m, wn) == common - oracle_lib.max_tract(a, b, m), t
