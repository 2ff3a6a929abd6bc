"""The block sums of the mixed-precision CG (Sum3 of csrc/fg_arith.h, the order of grid_reduce), compiled
for the host: pairs hi + lo of 1,024 threads against exact rational sums.  Bound: the three FP64
roundings of the final value and 2^-60 of the sum of magnitudes (the third word's roundings: 15 additions
of terms under 2^-47 of it, each rounded to 2^-24), where FP64 additions in the same order may lose
13 2^-53 of it."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "fempar_gb300", "csrc")
SOURCE = """
#include "fg_arith.h"
// n threads' pairs: 128 threads add every 128th, butterflies over 32 lanes, then over the four warps
extern "C" double block_sum(int n, const float* hi, const float* lo) {
  fg::Sum3 s[128], o[128];
  for (int t = 0; t < 128; ++t)
    for (int i = t; i < n; i += 128) s[t].add(hi[i], lo[i], 0.f);
  for (int off = 16; off > 0; off >>= 1) {
    for (int t = 0; t < 128; ++t) o[t] = s[t ^ off];
    for (int t = 0; t < 128; ++t) s[t].add(o[t].h, o[t].m, o[t].l);
  }
  fg::Sum3 w[4] = {s[0], s[32], s[64], s[96]}, y[4];
  for (int off = 1; off < 4; off <<= 1) {
    for (int t = 0; t < 4; ++t) y[t] = w[t ^ off];
    for (int t = 0; t < 4; ++t) w[t].add(y[t].h, y[t].m, y[t].l);
  }
  return w[0].value();
}
"""


@pytest.fixture(scope="module")
def block_sum(tmp_path_factory):
    d = tmp_path_factory.mktemp("sums")
    src, so = d / "sums.cpp", d / "sums.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)],
                   check=True)
    fn = ctypes.CDLL(str(so)).block_sum
    fn.restype = ctypes.c_double
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    return lambda hi, lo: fn(ctypes.c_int(len(hi)), ptr(hi), ptr(lo))


@pytest.mark.parametrize("signs", ["positive", "mixed", "cancelling"])
@pytest.mark.parametrize("spread", [0, 12, 40])
def test_block_sum(block_sum, signs, spread):
    rng = np.random.default_rng(spread)
    for n in (32, 96, 512, 1000, 1024):
        a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-spread - 1, spread + 1, n))
        b = np.ldexp(rng.uniform(1, 2, n), rng.integers(-spread - 1, spread + 1, n))
        if signs != "positive":
            a *= rng.choice([-1, 1], n)
        if signs == "cancelling":
            a[1::2], b[1::2] = -a[0::2], b[0::2] * (1 + 2.0 ** -20 * rng.standard_normal(n // 2))
        a, b = a.astype(np.float32), b.astype(np.float32)
        p = a.astype(np.float64) * b.astype(np.float64)  # exact
        hi = p.astype(np.float32)
        lo = (p - hi).astype(np.float32)  # exact: the product's 48 bits
        got = block_sum(hi, lo)
        exact = sum(Fraction(float(x)) + Fraction(float(y)) for x, y in zip(hi, lo))
        mag = sum(abs(Fraction(float(x))) for x in hi)
        assert abs(Fraction(got) - exact) <= 3 * Fraction(1, 2 ** 53) * abs(exact) + Fraction(1, 2 ** 60) * mag
