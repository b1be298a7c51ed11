"""The forms of the runs inside a word (glp_tract.h) as knn_tract_dist_kernel picks
them from a word's start, compiled for the host: each gives the oracle's
Haplotype::MaxTractLen, and haplotypes without long runs seldom end at the floor,
where a pair's words are gone through once more."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include "glp_tract.h"
// form 0, 1, 2: _inside32, _any, _long where `best` lets a word start with it
extern "C" uint32_t longest(const uint64_t *x, uint32_t wn, int form) {
  glp::OpenRun r{0, glp::kRunFloor};
  for (uint32_t w = 0; w < wn; ++w)
    for (int h = 0; h < 64; h += 32)
      glp::tract_extend32(r, (uint32_t)(x[w] >> h));
  for (uint32_t w = 0; w < wn; ++w) {
    const int f = form == 2 && r.best >= glp::kRunLong  ? 2
                  : form == 1 && r.best >= glp::kRunMid ? 1
                                                        : 0;
    for (int h = 0; h < 64; h += 32) {
      const uint32_t y = (uint32_t)(x[w] >> h);
      if (f == 2)
        glp::tract_inside32_long(r.best, y);
      else if (f == 1)
        glp::tract_inside32_any(r.best, y);
      else
        glp::tract_inside32(r.best, y);
    }
  }
  return r.best == glp::kRunFloor ? 0 : r.best;
}
'''


@pytest.fixture(scope="module")
def longest(tmp_path_factory):
    d = tmp_path_factory.mktemp("short")
    src, so = d / "short.cpp", d / "libshort.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-Wno-unknown-pragmas", "-I",
                    os.path.join(ROOT, "glphase_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = C.CDLL(str(so))
    L.longest.restype = C.c_uint32

    def run(differ, form):
        """differ: [pairs][sites] 0/1, whole words."""
        x = np.packbits(differ, axis=1, bitorder="little").view("<u8").astype(np.uint64)
        return np.array([L.longest(C.c_void_p(r.ctypes.data), C.c_uint32(len(r)), form)
                         for r in np.ascontiguousarray(x)])
    return run


def oracle(differ):
    best, run = np.zeros(len(differ), int), np.zeros(len(differ), int)
    for m in range(differ.shape[1]):
        run = np.where(differ[:, m], 0, run + 1)
        best = np.maximum(best, run)
    return best


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("p", [0.05, 0.2, 0.5, 0.8, 0.95])
def test_random_pairs(longest, form, p):
    d = (np.random.default_rng(int(100 * p)).random((3000, 192)) < p).astype(np.uint8)
    want = oracle(d)
    assert np.array_equal(longest(d, form), np.where(want > 1, want, 0))


@pytest.mark.parametrize("form", [0, 1, 2])
def test_one_run_of_every_length_and_place(longest, form):
    """Among disagreements, and beside a run that `best` already has from a word's
    edge: the test of each form lets no longer run pass."""
    rows = []
    for known in (0, 1, 2, 3, 6, 7, 8, 13, 14, 15, 16, 31):
        for n in range(1, 40):
            for at in range(0, 128 - n, 3):
                d = np.ones(192, np.uint8)
                d[at:at + n] = 0
                d[160 - known // 2:160 - known // 2 + known] = 0
                rows.append(d)
    d = np.array(rows)
    want = oracle(d)
    assert np.array_equal(longest(d, form), np.where(want > 1, want, 0))


@pytest.mark.parametrize("sites", [576, 1024])
def test_random_haplotypes_leave_the_floor(longest, sites):
    d = np.random.default_rng(sites).integers(0, 2, (5000, sites)).astype(np.uint8)
    assert (longest(d, 0) > 0).mean() > 0.999
