"""The device's last-bit arithmetic (csrc/fg_arith.h), compiled for the host.

quotient(s, d, 1/d) equals s / d bit for bit wherever quotient_exact(q, d) holds, over random operands
of every exponent, mantissas next to powers of two and to each other, subnormals, zeros, infinities and
NaN; and quotient_exact holds over the ordinary range (both operands within 2^+-40 in FP32, 2^+-400 in
FP64), so that the kernels' slow path is rare."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "fempar_gb300", "csrc")
SOURCE = """
#include "fg_arith.h"
extern "C" {
#define Q(T, NAME) \\
  void NAME(long n, const T* s, const T* d, T* q, unsigned char* exact) { \\
    for (long i = 0; i < n; ++i) { \\
      q[i] = fg::quotient(s[i], d[i], T(1) / d[i]); \\
      exact[i] = fg::quotient_exact(q[i], d[i]); \\
    } \\
  }
Q(float, quotient32)
Q(double, quotient64)
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("arith")
    src, so = d / "arith.cpp", d / "arith.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC, str(src), "-o", str(so)],
                   check=True)
    return ctypes.CDLL(str(so))


def quotients(lib, s, d):
    q, exact = np.empty_like(s), np.empty(len(s), dtype=np.uint8)
    fn = lib.quotient32 if s.dtype == np.float32 else lib.quotient64
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    fn(ctypes.c_long(len(s)), ptr(s), ptr(d), ptr(q), ptr(exact))
    return q, exact.astype(bool)


def operands(dtype, rng, n):
    bits, mant = (np.uint32, 23) if dtype == np.float32 else (np.uint64, 52)
    width = 32 if dtype == np.float32 else 64
    s = rng.integers(0, 2 ** width, n, dtype=bits).view(dtype)
    d = rng.integers(0, 2 ** width, n, dtype=bits).view(dtype)
    # mantissas at the edges, exponents at random
    edge = np.array([0, 1, 2, 2 ** mant - 1, 2 ** mant - 2, 2 ** (mant - 1), 2 ** (mant - 1) + 1], dtype=bits)
    exps = rng.integers(0, 2 ** (width - 1 - mant), (2, n), dtype=bits) << bits(mant)
    es = (exps[0] | rng.choice(edge, n)).view(dtype)
    ed = (exps[1] | rng.choice(edge, n)).view(dtype)
    near = (d.view(bits) + rng.integers(0, 4, n, dtype=bits)).view(dtype)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, np.finfo(dtype).max, np.finfo(dtype).tiny,
                        np.finfo(dtype).smallest_subnormal], dtype=dtype)
    sp, dp = (a.ravel() for a in np.meshgrid(special, special))
    return np.concatenate([s, es, s, es, near, sp]), np.concatenate([d, ed, ed, d, d, dp])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_quotient_is_the_division_where_it_says_so(lib, dtype):
    rng = np.random.default_rng(11)
    for _ in range(5):
        s, d = operands(dtype, rng, 400000)
        with np.errstate(all="ignore"):
            want = s / d
        q, exact = quotients(lib, s, d)
        tiny = np.finfo(dtype).smallest_subnormal
        same = (q == want) | ((q == 0) & (np.abs(want) <= tiny))
        assert same[exact].all()
        assert np.isfinite(q[exact]).all() and exact.mean() > 0.2


@pytest.mark.parametrize("dtype,range2", [(np.float32, 40), (np.float64, 400)])
def test_ordinary_operands_are_exact(lib, dtype, range2):
    rng = np.random.default_rng(12)
    n = 1000000
    draw = lambda: (np.ldexp(rng.uniform(1, 2, n), rng.integers(-range2, range2, n)) * rng.choice([-1, 1], n)).astype(dtype)
    s, d = draw(), draw()
    s[::7] = 0
    q, exact = quotients(lib, s, d)
    assert exact.all() and np.array_equal(q, s / d)
