"""The rule for a launch's speculation width (glp_width.h) compiled for the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include <chrono>
#include <cmath>
#include "glp_width.h"
extern "C" void steps(double a, double *out) {
  double s[glp::kWidths];
  glp::steps_a_round(a, s);
  for (int i = 0; i < glp::kWidths; ++i)
    out[i] = s[i];
}
extern "C" void shape(int rate, int *parent, int *accept) {
  const glp::SpecShape t = glp::make_spec_shape(rate);
  for (int i = 0; i < glp::kTeamNodes; ++i) {
    parent[i] = t.parent[i];
    accept[i] = t.accept[i];
  }
}
static double now() {
  return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}
// the least time of a pick, and of a thousand square roots of what came before
extern "C" void times(double *out) {
  const double resident[glp::kWidths] = {0, 152. * 128, 152. * 384, 152. * 384, 152. * 384,
                                         152. * 384, 152. * 384, 152. * 384};
  volatile unsigned sink = 0;
  volatile double root = 0;
  out[0] = out[1] = 1e9;
  for (int rep = 0; rep < 200; ++rep) {
    const double t0 = now();
    for (int i = 0; i < 10; ++i) {
      glp::WidthAsk ask;
      ask.rate = 0.001 * (1 + (i + rep) % 900);
      ask.samples = 3 + 97 * i;
      ask.sms = 152;
      ask.widest = 128;
      ask.resident = resident;
      sink = sink + glp::pick_lanes(ask);
    }
    const double t1 = now();
    double x = rep + 2.0;
    for (int i = 0; i < 1000; ++i)
      x = std::sqrt(x + 1.0);
    root = x;
    const double t2 = now();
    out[0] = std::min(out[0], (t1 - t0) / 10);
    out[1] = std::min(out[1], t2 - t1);
  }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("width")
    src, so = d / "width.cpp", d / "libwidth.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "glphase_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = C.CDLL(str(so))
    L.steps.argtypes = [C.c_double, C.c_void_p]
    return L


@pytest.mark.parametrize("a", [0.0, 1e-3, 0.03, 0.12, 0.35, 0.5, 0.77, 0.96, 0.99, 1.0])
def test_steps(lib, a):
    """The sum of the nodes' chances, each the product along its own path."""
    rate = min(int(a * 16 + 0.5), 16)
    parent, accept = (C.c_int * 64)(), (C.c_int * 64)()
    lib.shape(rate, parent, accept)
    got = np.zeros(8)
    lib.steps(a, got.ctypes.data)
    for i in range(1, 8):
        n = 2 ** (i - 1)
        if n < 8:
            want = sum((1 - a) ** k for k in range(n))
        else:
            want = 0.0
            for k in range(n):
                p, v = 1.0, k
                while v:
                    p *= a if accept[v] else 1 - a
                    v = parent[v]
                want += p
        assert abs(got[i] - want) < 1e-9 * want, i


def test_host_time(lib):
    """A pick runs before every launch: it may take as long as 1,000 dependent square
    roots (7 us here; it takes 0.3, and took 14 with a power of the rate for every node
    of every width, beside 85 for a whole generation of three samples and sites)."""
    t = (C.c_double * 2)()
    lib.times(t)
    assert t[0] < t[1], (t[0], t[1])
