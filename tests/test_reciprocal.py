"""The FP64 pivots' reciprocal (uchol_check_reciprocal) against 1 / p in integers, and against IEEE division where it divides."""
from fractions import Fraction

import numpy as np
import pytest

from magla_gb300 import _native
from magla_gb300.errors import raise_for_status

pytestmark = pytest.mark.gpu


def reciprocal(p):
    p = np.ascontiguousarray(p, np.float64)
    out = np.zeros_like(p)
    lib = _native.gpu()
    raise_for_status(lib.uchol_check_reciprocal(len(p), p.ctypes.data, out.ctypes.data), lib.uchol_last_error())
    return out


def ulps(p, x):
    """|x - 1 / p| in units of x's last place."""
    e = int(np.frexp(x)[1]) - 53
    return float(abs(Fraction(float(x)) - 1 / Fraction(float(p))) / Fraction(2) ** e)


def test_bound(gpu_lib):
    rng = np.random.default_rng(0)
    one = 1.0 + np.arange(64) * 2.0 ** -52
    steps = 1.0 + (np.arange(1, 65) * 2.0 ** -6) - 2.0 ** -52                # ends of the leading bits' intervals, past 2^-23
    low = 1.0 + rng.integers(0, 1 << 23, 2000) * 2.0 ** -23 + (2.0 ** -23 - 2.0 ** -52)   # all bits that FP32 leaves out
    s = np.concatenate([one, 2.0 - np.arange(1, 65) * 2.0 ** -52, steps, low, rng.uniform(1.0, 2.0, 4000)])
    p = np.ldexp(s, rng.integers(-120, 121, len(s)))
    p = np.concatenate([p, np.ldexp(s[:400], -120), np.ldexp(s[:400], 120)])
    x = reciprocal(p)
    assert max(ulps(a, b) for a, b in zip(p, x)) <= 0.5003


def test_divided_arguments(gpu_lib):
    rng = np.random.default_rng(1)
    s = np.concatenate([rng.uniform(1.0, 2.0, 200), [1.0, 2.0 - 2.0 ** -52]])
    p = np.concatenate([np.ldexp(s, k) for k in (-1022, -500, -121, 121, 500, 1023)] +
                       [-np.ldexp(s, k) for k in (-121, -120, 0, 120)] +
                       [[0.0, -0.0, 5e-324, 2.0 ** -1030, np.inf, -np.inf, np.nan]])
    with np.errstate(all="ignore"):
        ref = 1.0 / p
    assert np.array_equal(reciprocal(p), ref, equal_nan=True)
    assert np.array_equal(np.signbit(reciprocal(p))[:-1], np.signbit(ref)[:-1])
