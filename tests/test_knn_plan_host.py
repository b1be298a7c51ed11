"""The plan of a neighbour table (glp_knn_plan.h) compiled for the host: its memory
within the limit, every sample and operand row covered, and, against a fake device
that has so many bytes left, the widest plan that fits -- in 256 MB, which any table
was built in before whole panels were held, always one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include "glp_knn_plan.h"
using glp::KnnPlan;
static void put(const KnnPlan &p, unsigned long long *o) {
  o[0] = p.whole; o[1] = p.sym; o[2] = p.pitch; o[3] = p.chunk; o[4] = p.bytes; o[5] = p.slab;
  o[6] = p.dist_bytes(); o[7] = p.operand_bytes();
}
extern "C" void plan(unsigned H, unsigned S, int tract, unsigned long long limit,
                     unsigned long long *o) {
  put(glp::knn_plan(H, S, tract != 0, limit), o);
}
// a device with `room` bytes; returns the status, o[8] the attempts
extern "C" int fit(unsigned H, unsigned S, int tract, unsigned long long room, int other,
                   unsigned long long *o) {
  KnnPlan p;
  o[8] = 0;
  const int rc = glp::knn_fitting_plan(H, S, tract != 0, ~(size_t)0, 3, [&](const KnnPlan &q) {
    ++o[8];
    return other ? other : q.total() <= room ? 0 : 3;
  }, &p);
  put(p, o);
  return rc;
}
'''
MB = 1 << 20
SIZES = [(4, 1), (60, 64), (254, 65534), (2000, 65534), (5000, 1024), (20000, 4096), (23000, 500),
         (24002, 64), (30000, 65534), (50000, 64), (50000, 22000), (50000, 65534)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, so = d / "plan.cpp", d / "libplan.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "glphase_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    return C.CDLL(str(so))


def call(f, *args):
    o = (C.c_ulonglong * 9)()
    rc = f(*args, o)
    keys = ("whole", "sym", "pitch", "chunk", "bytes", "slab", "dist", "ops", "tries")
    return rc, dict(zip(keys, [int(x) for x in o]))


@pytest.mark.parametrize("tract", [0, 1])
@pytest.mark.parametrize("H,S", SIZES)
def test_every_limit(lib, H, S, tract):
    for limit in (0, 1 * MB, 30 * MB, 256 * MB, 700 * MB, 2048 * MB, 2**64 - 1):
        _, p = call(lib.plan, C.c_uint(H), C.c_uint(S), tract, C.c_ulonglong(limit))
        assert p["pitch"] >= H and p["pitch"] % 128 == 0 and p["bytes"] >= S
        assert 1 <= p["chunk"] <= H // 2
        if tract:
            assert p["ops"] == 0
        else:
            assert p["ops"] == (H * p["bytes"] if p["whole"] else 2 * p["slab"] * p["bytes"])
            assert p["whole"] or (p["slab"] >= 256 and p["slab"] % 256 == 0)
            assert p["slab"] == H or not p["whole"]
        if p["sym"]:
            assert p["chunk"] == H // 2 and (p["whole"] or tract)
        least = 4 * min(64, H // 2) * p["pitch"] + (0 if tract else 512 * p["bytes"])
        assert p["dist"] + p["ops"] <= max(limit, least)
        assert p["dist"] <= 1024 * MB and p["ops"] <= max(1024 * MB, 512 * p["bytes"])


@pytest.mark.parametrize("tract", [0, 1])
@pytest.mark.parametrize("H,S", SIZES)
def test_what_fits(lib, H, S, tract):
    _, widest = call(lib.plan, C.c_uint(H), C.c_uint(S), tract, C.c_ulonglong(2**64 - 1))
    for room in (2048 * MB, 1200 * MB, 700 * MB, 256 * MB):
        rc, p = call(lib.fit, C.c_uint(H), C.c_uint(S), tract, C.c_ulonglong(room), 0)
        assert rc == 0 and p["dist"] + p["ops"] <= room
        if widest["dist"] + widest["ops"] <= room:
            assert p["tries"] == 1 and p["dist"] == widest["dist"]
    rc, p = call(lib.fit, C.c_uint(H), C.c_uint(S), tract, C.c_ulonglong(0), 0)
    assert rc == 3 and p["tries"] <= 3          # no memory at all: the error comes back
    rc, p = call(lib.fit, C.c_uint(H), C.c_uint(S), tract, C.c_ulonglong(0), 5)
    assert rc == 5 and p["tries"] == 1          # and another error straight away


def test_fake_sizes_of_the_listed_table(lib):
    """20,000 x 4,096: 886 MB; with less, in pieces."""
    rc, p = call(lib.fit, C.c_uint(20000), C.c_uint(4096), 0, C.c_ulonglong(900 * MB), 0)
    assert rc == 0 and p["sym"] and 840 * MB < p["dist"] + p["ops"] < 890 * MB
    rc, p = call(lib.fit, C.c_uint(20000), C.c_uint(4096), 0, C.c_ulonglong(800 * MB), 0)
    assert rc == 0 and not p["sym"] and p["tries"] == 2
