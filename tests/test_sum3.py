"""The three-float sum of the FP32 dots (csrc/tg_sum.h) against exact rational arithmetic.

Bound: every addition rounds the third float alone, whose size is at most depth * 2^-48 of the
sum of magnitudes S; depth additions on a path lose depth^2 2^-72 S.  Paths here are below 32
additions: 2^-62 S, against FP64's 2^-53 an addition.
"""

import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <vector>
#include "tg_sum.h"
using tg::Sum3;
// n pairs (hi, lo): lanes of 32 add in turn, then the tree of a warp
extern "C" double tree(const float* hi, const float* lo, int n, float* out) {
  std::vector<Sum3> w(32, Sum3::of(0.f, 0.f));
  for (int i = 0; i < n; ++i) {
    if (i & 32) w[i & 31].add(hi[i], lo[i]);
    else w[i & 31].add(Sum3::of(hi[i], lo[i]));
  }
  for (int o = 16; o > 0; o >>= 1)
    for (int l = 0; l < o; ++l) w[l].add(w[l + o]);
  w[0].normalize();
  out[0] = w[0].s; out[1] = w[0].c; out[2] = w[0].cc;
  return w[0].value();
}
extern "C" void split(double v, float* out) {
  const Sum3 t = Sum3::of(v);
  out[0] = t.s; out[1] = t.c; out[2] = t.cc;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sum3")
    src, so = d / "sum3.cpp", d / "sum3.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "tatva_gb300", "csrc"), str(src), "-o", str(so)],
                   check=True)
    L = ctypes.CDLL(str(so))
    L.tree.restype = ctypes.c_double
    return L


def _floats(p):
    return p.ctypes.data_as(ctypes.POINTER(ctypes.c_float))


@pytest.mark.parametrize("n", [1, 31, 64, 801])
@pytest.mark.parametrize("signed", [False, True])
def test_sums_lose_less_than_fp64(lib, n, signed):
    rng = np.random.default_rng(n)
    hi = np.exp(rng.normal(0, 6, n)).astype(np.float32)
    if signed:
        hi *= np.where(rng.random(n) < 0.5, -1, 1).astype(np.float32)
    lo = (hi * rng.uniform(-2.0**-25, 2.0**-25, n)).astype(np.float32)
    out = np.zeros(3, np.float32)
    value = lib.tree(_floats(hi), _floats(lo), n, _floats(out))
    exact = sum((Fraction(float(a)) + Fraction(float(b)) for a, b in zip(hi, lo)), Fraction(0))
    size = sum(abs(Fraction(float(a))) + abs(Fraction(float(b))) for a, b in zip(hi, lo))
    got = sum(Fraction(float(t)) for t in out)
    assert abs(got - exact) <= size * Fraction(2) ** -62
    # FP64 rounds the result once
    assert abs(Fraction(value) - got) <= abs(got) * Fraction(2) ** -52
    assert abs(out[1]) <= abs(out[0]) * 2.0**-24 and out[0] == np.float32(value)


@pytest.mark.parametrize("v", [0.0, 1.0, -np.pi, 1e-30, 3.3e38, 1 + 2.0**-52])
def test_fp64_values_split_exactly(lib, v):
    out = np.zeros(3, np.float32)
    lib.split(ctypes.c_double(v), _floats(out))
    assert sum(Fraction(float(t)) for t in out) == Fraction(v)
