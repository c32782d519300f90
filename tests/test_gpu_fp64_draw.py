"""The FP64 chain's latent draw by itself against 40-digit values, and the quotients
by reciprocal and the reciprocal square root that the draws of the coefficients and
of Omega use.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_draw_against_40_digits():
    mpmath = pytest.importorskip("mpmath")
    from bsglmm_gb300 import _lib
    rng = np.random.default_rng(3)
    # all rows of the Mills ratio's table and their edges, both tails, the largest
    # and smallest words
    a = np.concatenate([rng.uniform(-12, 5, 3000), np.arange(-96, 41) / 8,
                        np.arange(-97, 40) / 8 + 0.0625, np.nextafter(np.arange(-97, 40) / 8
                                                                      + 0.0625, 99),
                        [5.0, 4.999999, 0.0, -0.0, -5e-324, -36.99, -20.0]])
    k = rng.integers(0, 1 << 32, a.size, dtype=np.uint64).astype(np.uint32)
    edge = np.array([0, 1, 0xFFFFFFFF, 0xFFFFFFFE, 0x7FFFFFFF, 0x80000000], np.uint32)
    rows = a[3000:]
    a = np.concatenate([a, np.tile(rows, edge.size)])
    k = np.concatenate([k, np.repeat(edge, rows.size)])
    t = np.empty_like(a)
    L = _lib.lib()
    p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert L.bsg_selftest_draw64(0, a.size, p(a), p(k), p(t)) == 0
    err = np.empty_like(a)
    with mpmath.workdps(40):
        r2 = mpmath.sqrt(2)
        for i in range(a.size):
            uc = 1 - (mpmath.mpf(int(k[i])) + 0.5) / 2 ** 32
            x = mpmath.mpf(float(t[i]))
            tail = mpmath.erfc(mpmath.mpf(float(a[i])) / r2) / 2 * uc
            phi = mpmath.exp(-x * x / 2) / mpmath.sqrt(2 * mpmath.pi)
            err[i] = float((mpmath.erfc(x / r2) / 2 - tail) / phi)
    err /= np.maximum(1.0, np.abs(t))
    print(f"rms {np.sqrt(np.mean(err[:3000] ** 2)):.2e}, largest {np.abs(err).max():.2e}")
    # some eight roundings of 1.1e-16 of a tail, times the Mills ratio's 1.25
    assert np.abs(err).max() < 1.2e-15
    assert L.bsg_selftest_draw64(0, 0, p(a), p(k), p(t)) != 0


def test_quotients_and_reciprocal_square_roots():
    from bsglmm_gb300 import _lib
    bad, err = C.c_int64(-1), C.c_double(-1)
    assert _lib.lib().bsg_selftest_quotients(0, 1 << 28, 0x51EE_D002, C.byref(bad),
                                             C.byref(err)) == 0
    print(f"{bad.value} quotients of 2^28 differ, reciprocal square root {err.value:.2f} x 2^-53")
    assert bad.value == 0
    # the remainder of the third-order step, 5/16 (2^-22)^3, and three roundings
    assert 0 < err.value < 3.1
