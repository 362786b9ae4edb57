"""The arithmetic of the persistent PCG kernel's grid sums (grid_scale.h) on
the host: partial sums of blocks -> limbs -> sum, with the repeats at another
scale that the kernel makes.  The number of repeats is bounded whatever the
partials, cancelling ones among them, and the sum is as good as an FP64 sum.

Error bound: a limb sum beyond 2^53 is rounded to FP64 (2^-53 of the sum of the
sizes), the three are added (2^-51 of the result), and at the scale where a sum
is taken what is dropped lies below 2^-56 of the result or 2^-58 of the largest
partial."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

SOURCE = r"""
#include "grid_scale.h"
using namespace fastgpu;
// the sum of n partials as grid_sum forms it; the repeats it took, or -1 beyond cap
extern "C" int grid_sum_host(int n, const double *x, double ref, int cap, double *out) {
  SumScale s = sum_scale(ref);
  for (int rep = 0; rep <= cap; rep++) {
    int64_t w[3] = {0, 0, 0};
    for (int i = 0; i < n; i++)
      for (int l = 0; l < 3; l++) w[l] += sum_limb(x[i], s.e, l);
    double d[3];
    for (int l = 0; l < 3; l++) d[l] = scale2((double)w[l], limb_exponent(s.e, l));
    double res = d[0] + (d[1] + d[2]);
    const bool again = sum_again(s, w[0] >= kSumMarked, res);
    *out = res;
    if (!again) return rep;
  }
  return -1;
}
"""


@pytest.fixture(scope="module")
def grid_sum(tmp_path_factory):
    d = tmp_path_factory.mktemp("gridsum")
    src, lib = d / "gridsum.cpp", d / "gridsum.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "fast_b200", "csrc"), "-o", str(lib), str(src)], check=True)
    f = ctypes.CDLL(str(lib)).grid_sum_host
    f.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_double), ctypes.c_double, ctypes.c_int,
                  ctypes.POINTER(ctypes.c_double)]

    def call(x, ref):
        a = np.ascontiguousarray(x, dtype=np.float64)
        out = ctypes.c_double()
        n = f(len(a), a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), ref, 200, ctypes.byref(out))
        return n, out.value
    return call


MAX_REPEATS = 80


def check(call, x, ref, most=MAX_REPEATS):
    n, s = call(x, ref)
    assert 0 <= n <= most, f"{n} repeats"
    ex = sum((Fraction(float(v)) for v in x), Fraction(0))
    size = sum((abs(Fraction(float(v))) for v in x), Fraction(0))
    assert abs(Fraction(s) - ex) <= abs(ex) * Fraction(1, 2**50) + size * Fraction(1, 2**52)
    return n, s


def block(v, n=148):
    return np.concatenate([np.asarray(v, float), np.zeros(n - len(v))])


@pytest.mark.parametrize("x", [[1.0, -1.0], [1.0, -1.0 + 2.0**-30], [1.0, -1.0 - 2.0**-30], [3.0, -1.0, -2.0],
                               [1.0, -1.0 + 2.0**-53], [1e200, -1e200], [1e-200, -1e-200],
                               [1.0, 2.0**-100, -1.0], [0.1, 0.2, -0.3]])
@pytest.mark.parametrize("ref", [1.0, -1.0, 0.0, 1e-30, 1e30, 1e-300, 1e299, math.nan, math.inf])
def test_cancelling_partials_end(grid_sum, x, ref):
    check(grid_sum, block(x), ref)


def test_random_partials(grid_sum):
    rng = np.random.default_rng(7)
    for _ in range(3000):
        n = int(rng.integers(1, 149))
        x = rng.standard_normal(n) * 2.0 ** rng.integers(-60, 61, size=n) * 2.0 ** float(rng.integers(-400, 401))
        if rng.random() < 0.5:
            x[-1] = 0.0
            x[-1] = -math.fsum(x) * (1.0 + rng.choice([0.0, 1e-9, 1e-16]))
        check(grid_sum, x, float(rng.choice([abs(x).max(), 1.0, 0.0, abs(x).max() * 1e-40])))


def test_ordinary_sums_are_formed_once(grid_sum):
    """Positive partials within 2^40 of the last value: no repeat."""
    rng = np.random.default_rng(8)
    for _ in range(500):
        x = rng.random(148) * 2.0 ** float(rng.integers(-200, 200))
        ref = math.fsum(x) * 10.0 ** rng.uniform(-6, 6)
        check(grid_sum, x, ref, most=0)


@pytest.mark.parametrize("x,ref", [([0.0], 1.0), ([0.0], 1e-300), ([1e-290], 1.0), ([5e-150, -5e-150], 1e250),
                                   ([1.7e308], 1.0), ([1e300, 1e300], 0.0), ([1e-300, 3e-305], 1e-300)])
def test_ends_of_the_range(grid_sum, x, ref):
    check(grid_sum, block(x), ref)


@pytest.mark.parametrize("v", [math.inf, -math.inf, math.nan])
def test_not_finite(grid_sum, v):
    n, s = grid_sum(block([1.0, v]), 1.0)
    assert 0 <= n <= MAX_REPEATS and not math.isfinite(s)
