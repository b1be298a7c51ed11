"""The product of an evaluation's halves (glp_join.h: pairs of floats, as log_dot
runs them on the device) compiled for the host, against the binary64 product: the
same mantissa and exponent, bit for bit, wherever it claims a result -- on random
states of a blocked pass, on sums placed around the middle between two floats and
around powers of two, and outside its range, where it must claim none."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include "glp_join.h"
extern "C" void run(const float *x, const float *y, uint32_t n, float *m, int *e, uint8_t *ok) {
  for (uint32_t i = 0; i < n; ++i) {
    const float *a = x + 4 * i, *b = y + 4 * i;
    ok[i] = glp::join_product(a[0], a[1], a[2], a[3], b[0], b[1], b[2], b[3], m[i], e[i]);
  }
}
'''


@pytest.fixture(scope="module")
def join(tmp_path_factory):
    d = tmp_path_factory.mktemp("join")
    src, so = d / "join.cpp", d / "libjoin.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "glphase_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = C.CDLL(str(so))

    def run(x, y):
        x, y = np.ascontiguousarray(x, np.float32), np.ascontiguousarray(y, np.float32)
        n = len(x)
        m, e, ok = np.zeros(n, np.float32), np.zeros(n, np.int32), np.zeros(n, np.uint8)
        L.run(*(C.c_void_p(a.ctypes.data) for a in (x, y)), C.c_uint32(n),
              *(C.c_void_p(a.ctypes.data) for a in (m, e, ok)))
        return m, e, ok.astype(bool)
    return run


def binary64(x, y):
    """The product in binary64 (each of the four is exact there), its mantissa in
    [1, 2) rounded to binary32, and its exponent."""
    p = x.astype(np.float64) * y.astype(np.float64)
    dot = ((p[:, 0] + p[:, 1]) + p[:, 2]) + p[:, 3]
    m, e = np.frexp(dot)
    return (2 * m).astype(np.float32), e - 1


def check(join, x, y, claimed):
    m, e, ok = join(x, y)
    wm, we = binary64(x, y)
    assert np.array_equal(m[ok].view(np.uint32), wm[ok].view(np.uint32))
    assert np.array_equal(e[ok], we[ok])
    assert ok.mean() >= claimed
    return ok


def states(rng, n, spread):
    """Four states of one sum, as a block leaves them."""
    v = np.exp(rng.uniform(-spread, 0, (n, 4)))
    return (v / v.sum(axis=1, keepdims=True) * 2.0**62 * rng.uniform(1, 2, (n, 1))).astype(np.float32)


@pytest.mark.parametrize("spread", [0.1, 3.0, 20.0, 60.0])
def test_random_states(join, spread):
    rng = np.random.default_rng(int(10 * spread))
    check(join, states(rng, 500000, spread), states(rng, 500000, spread), 1 - 2.0**-12)


def test_sums_next_to_the_middle_of_two_floats(join):
    """hi + half a unit +- 2^-k units, the small part in one product or in the
    binary32 rounding of two others."""
    rng = np.random.default_rng(1)
    rows = []
    for k in range(2, 34):
        for _ in range(200):
            hi = np.float32(rng.integers(2**23, 2**24))     # one product, unit 1
            up = np.float32(2.0**-k)
            half = np.float32(0.5)
            big = rng.integers(2**20, 2**23)                # another, that makes s inexact
            rows.append([hi, half, up, 0.0])
            rows.append([hi, half - up if k < 24 else half, 0.0, up / 2])
            rows.append([hi, float(big) + 0.25, 0.25, up])
            rows.append([up, hi, 0.25, float(big) + 0.25])
    x = np.array(rows, np.float32) * np.float32(2.0**40)
    y = np.full_like(x, 2.0**20)
    check(join, x, y, 0.3)
    # products that are not powers of two apart: (a + b) (a - b) forms with long tails
    a = rng.integers(2**23, 2**24, (200000, 4)).astype(np.float32)
    b = rng.integers(2**23, 2**24, (200000, 4)).astype(np.float32)
    a[:, 1:] *= np.float32(2.0) ** rng.integers(-30, -22, (200000, 3)).astype(np.float32)
    check(join, a * np.float32(2.0**20), b, 1 - 2.0**-9)


def test_powers_of_two_are_left_to_binary64(join):
    x = np.zeros((4, 4), np.float32)
    x[:, 0] = 2.0**60
    x[1, 1] = 2.0**20      # just above: rounds down to the power
    x[2, 0] = np.nextafter(np.float32(2.0**60), np.float32(0))
    x[2, 1] = 2.0**35      # just below: rounds up to it
    x[3, :] = 2.0**58
    assert not join(x, np.full_like(x, 2.0**10))[2].any()


@pytest.mark.parametrize("f,g", [(2.0**-70, 2.0**-70), (2.0**-40, 2.0**-25), (2.0**64, 2.0**64),
                                 (0.0, 1.0), (np.inf, 1.0), (np.nan, 1.0), (1e-40, 1e-3),
                                 (-1.0, 1.0)])
def test_outside_its_range(join, f, g):
    x = np.full((3, 4), f, np.float32) * np.float32([1.1, 1.3, 1.7])[:, None]
    y = np.full((3, 4), g, np.float32)
    assert not join(x, y)[2].any()
