"""The quotient from a kept reciprocal: csrc/div_by.cuh itself, compiled for the host
(with a stand-in for the one device intrinsic it uses), against the division.

Bit for bit where its header says so: normal quotients of operands whose residual
cannot underflow (|a| from 2^-900, b and 1 / b normal).  Zero, infinite and NaN
quotients, of zero, infinite or NaN operands too, equal the division's with their
sign.  A subnormal quotient is the estimate a y, whose factor y = RN(1 / b) and whose
product are each rounded once: within one unit 2^-1074 of the division's, which is
rounded once itself."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from wavetrisk_hydrostatic_b200 import build

SHIM = r"""
#include <cmath>
#include <cstring>
static inline int __double2hiint(double x) { long long b; std::memcpy(&b, &x, 8); return (int)(b >> 32); }
using std::fma;
#include "div_by.cuh"
extern "C" void quotients(const double* a, const double* b, double* q, double* d, long n) {
  for (long k = 0; k < n; ++k) {
    q[k] = wtk::div_by(a[k], b[k], 1.0 / b[k]);
    d[k] = a[k] / b[k];
  }
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    d = tmp_path_factory.mktemp("div_by")
    src, lib = d / "shim.cpp", d / "libdiv_by.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-Wno-attributes", "-fPIC", "-shared",
                    "-I", build.CSRC, "-I", os.path.join(build.CUDA_HOME, "include"), str(src), "-o", str(lib)],
                   check=True)
    f = ctypes.CDLL(str(lib)).quotients
    p = np.ctypeslib.ndpointer(np.float64, flags="C")
    f.argtypes = [p, p, p, p, ctypes.c_long]

    def run(a, b):
        a, b = np.broadcast_arrays(np.asarray(a, float), np.asarray(b, float))
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        q, d = np.empty_like(a), np.empty_like(a)
        f(a, b, q, d, a.size)
        return q, d

    return run


def _mantissas(kind, n, rng):
    if kind == "near2":    # just below 2: the reciprocal's hardest
        return 2.0 - rng.integers(1, 64, n) * 2.0 ** -52
    if kind == "near1":
        return 1.0 + rng.integers(0, 64, n) * 2.0 ** -52
    if kind == "short":    # quotients that are exact or halfway
        return 1.0 + rng.integers(0, 2 ** 12, n) * 2.0 ** -12
    return 1.0 + rng.integers(0, 2 ** 52, n) * 2.0 ** -52


@pytest.mark.parametrize("kb", ["any", "near2", "near1", "short"])
@pytest.mark.parametrize("ka", ["any", "near2", "near1", "short"])
def test_normal_quotients_are_the_divisions(quotients, ka, kb):
    rng = np.random.default_rng(len(ka) * 16 + len(kb))
    n = 200000
    a = np.ldexp(_mantissas(ka, n, rng) * rng.choice([-1.0, 1.0], n), rng.integers(-900, 1000, n))
    b = np.ldexp(_mantissas(kb, n, rng) * rng.choice([-1.0, 1.0], n), rng.integers(-1000, 1000, n))
    q, d = quotients(a, b)
    normal = np.isfinite(d) & (np.abs(d) >= 2.0 ** -1021) & (np.abs(d) < 2.0 ** 1023)
    assert normal.sum() > n // 2
    assert np.array_equal(q[normal], d[normal])


def test_zero_infinite_and_nan(quotients):
    v = np.array([0.0, -0.0, 1.0, -3.0, 1e300, -1e-300, np.inf, -np.inf, np.nan])
    a, b = np.repeat(v, v.size), np.tile(v, v.size)
    with np.errstate(all="ignore"):
        q, d = quotients(a, b)
    special = np.isnan(d) | np.isinf(d) | (d == 0)
    assert special.sum() > 40
    assert np.array_equal(q[special], d[special], equal_nan=True)
    sign = special & ~np.isnan(d)
    assert np.array_equal(np.signbit(q[sign]), np.signbit(d[sign]))


def test_subnormal_and_overflowing_quotients(quotients):
    rng = np.random.default_rng(5)
    n = 200000
    a = np.ldexp(_mantissas("any", n, rng), rng.integers(-900, -600, n))
    b = np.ldexp(_mantissas("any", n, rng), rng.integers(100, 500, n))
    q, d = quotients(a, b)
    sub = np.abs(d) < 2.0 ** -1022
    assert sub.sum() > n // 50
    assert np.abs(q[sub] - d[sub]).max() <= 2.0 ** -1074
    q, d = quotients(np.ldexp(1.5, np.arange(900, 1023)), np.ldexp(1.25, -np.arange(200, 323)))
    assert np.isinf(d).all() and np.array_equal(q, d)
