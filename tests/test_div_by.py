"""The quotient from a kept reciprocal (div_by of csrc/trisk_read.cuh) against the
division, bit for bit: its operations, in this order, with the C library's fma."""
import ctypes
import ctypes.util

import numpy as np
import pytest

_libm = ctypes.CDLL(ctypes.util.find_library("m"))
_libm.fma.restype = ctypes.c_double
_libm.fma.argtypes = [ctypes.c_double] * 3
fma = _libm.fma


def div_by(a, b, y):
    q0 = float(np.float64(a) * np.float64(y))
    q1 = fma(fma(-b, q0, a), y, q0)
    q2 = fma(fma(-b, q1, a), y, q1)
    return q2 if np.isfinite(q0) and abs(q0) >= 2.0 ** -1022 else q0


def _values(kind, n, rng):
    m = 1.0 + rng.integers(0, 2 ** 52, n).astype(np.float64) * 2.0 ** -52
    if kind == "ones":  # mantissas next to 2: the reciprocal's hardest
        m = 2.0 - rng.integers(1, 64, n).astype(np.float64) * 2.0 ** -52
    if kind == "short":  # quotients that are exact or halfway
        m = 1.0 + rng.integers(0, 2 ** 12, n).astype(np.float64) * 2.0 ** -12
    return np.ldexp(m * rng.choice([-1.0, 1.0], n), rng.integers(-300, 300, n))


@pytest.mark.parametrize("ka", ["any", "ones", "short"])
@pytest.mark.parametrize("kb", ["any", "ones", "short"])
def test_quotient_is_the_divisions(ka, kb):
    rng = np.random.default_rng(len(ka) * 7 + len(kb))
    a, b = _values(ka, 4000, rng), np.abs(_values(kb, 4000, rng))
    for x, z in zip(a.tolist(), b.tolist()):
        assert div_by(x, z, 1.0 / z) == x / z


def test_special_values():
    with np.errstate(all="ignore"):
        for b in (1.0, 3.0, 1000.0, np.inf):
            for a in (0.0, -0.0, np.inf, -np.inf, np.nan):
                got, want = div_by(a, b, float(np.float64(1.0) / np.float64(b))), np.float64(a) / np.float64(b)
                assert np.array_equal([got], [want], equal_nan=True) and (np.isnan(want) or np.signbit(got) == np.signbit(want))
