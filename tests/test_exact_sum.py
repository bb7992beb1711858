"""Order-free sums (csrc/exact_sum.h): the fixed-point accumulator, compiled for the host, against exact rational
sums rounded once, for terms of any size, sign and order."""
import ctypes
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "realmolecule_b200", "csrc")

SRC = r"""
#include "exact_sum.h"
using namespace rq;
extern "C" double exact_sum(const double* x, long long n) {
  long long w[kExWords] = {}, p[3];
  for (long long q = 0; q < n; ++q) {
    const int i = exact_split(x[q], p);
    if (i == kExFlags) w[i] |= p[0];
    else for (int k = 0; k < 3; ++k) w[i + k] += p[k];
  }
  int first = 0, last = 0;  // the limbs that are not 0, as the kernels find them
  while (first < kExLimbs - 1 && !w[first]) ++first;
  for (int i = 0; i < kExLimbs; ++i) if (w[i]) last = i;
  if (!w[first]) first = 0;
  return exact_round([&](int i) { return w[i]; }, first, last, w[kExFlags]);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("exact")
    (d / "t.cpp").write_text(SRC)
    subprocess.run([cc, "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    l = ctypes.CDLL(str(d / "t.so"))
    l.exact_sum.restype, l.exact_sum.argtypes = ctypes.c_double, [ctypes.c_void_p, ctypes.c_longlong]

    def total(x):
        a = np.array(x, np.float64)
        return l.exact_sum(a.ctypes.data, len(a))

    return total


def _rounded(x):
    s = sum(map(Fraction, x), Fraction(0))
    try:
        return float(s)
    except OverflowError:
        return math.inf if s > 0 else -math.inf


@pytest.mark.parametrize("spread", [0, 3, 60, 700])
def test_sum_is_the_rounded_exact_sum(lib, spread):
    rng = np.random.default_rng(spread)
    for t in range(1500):
        n = int(rng.integers(0, 30))
        e = np.clip(rng.uniform(-1074, 1024) + rng.uniform(-spread, spread, n), -1074, 1024).astype(int)
        x = [math.ldexp(float(rng.choice((-1, 1)) * rng.uniform(0.5, 1)), int(q)) for q in e]
        if t % 3 == 0:
            x = [abs(v) for v in x]
        if t % 5 == 0 and n > 2:
            x += [-v for v in x[1:]]  # cancels down to one term
        assert lib(x) == _rounded(x)
        assert lib(x) == lib(list(rng.permutation(x)))


def test_edges(lib):
    inf, nan = math.inf, math.nan
    for x in ([], [0.0], [-0.0], [5e-324] * 3, [-5e-324], [2.0 ** 53, 1.0], [2.0 ** 53, 1.0, 5e-324], [2.0 ** 53, 3.0],
              [1e308] * 9, [-1e308] * 9, [1e308] * 9 + [-1e308] * 8, [1.7976931348623157e308, 2.0 ** 969],
              [1.7976931348623157e308, 2.0 ** 970], [1e-320] * 1000):
        assert lib(x) == _rounded(x)
    assert lib([inf, 1.0]) == inf and lib([1.0, -inf]) == -inf
    assert math.isnan(lib([inf, -inf])) and math.isnan(lib([nan, 1.0])) and math.isnan(lib([nan, inf]))
