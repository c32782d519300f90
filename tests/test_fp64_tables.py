"""CPU check of the FP64 draw's tables (bsglmm_gb300/csrc/bsg_mills_table.h) against
40-digit values: every row of the Mills ratio over its interval, every power of two.
"""
from __future__ import annotations

import re
from pathlib import Path

import pytest

mpmath = pytest.importorskip("mpmath")

HDR = Path(__file__).resolve().parents[1] / "bsglmm_gb300" / "csrc" / "bsg_mills_table.h"


def _table(name):
    text = HDR.read_text()
    body = text[text.index(name):]
    body = body[body.index("{") + 1:body.index("}")]
    return [float.fromhex(x) if "0x" in x else float(x)
            for x in re.findall(r"[-+]?0x[0-9a-fA-F.]+p[-+]?\d+|[-+]?\d+\.\d+e[-+]?\d+", body)]


def test_mills_rows():
    c = _table("kMillsTable")
    rows, coef = 89, 9
    assert len(c) == rows * coef
    worst = 0
    with mpmath.workdps(40):
        for j in range(rows):
            # |h| <= 1/16 and a little over, as the rows are picked in FP32
            for i in range(-8, 9):
                h = mpmath.mpf(i) / 128 * (1 + mpmath.mpf(2) ** -20)
                x = mpmath.mpf(j) / 8 + h
                r = mpmath.sqrt(mpmath.pi / 2) * mpmath.exp(x * x / 2) * mpmath.erfc(
                    x / mpmath.sqrt(2))
                got = mpmath.polyval([mpmath.mpf(v) for v in c[j * coef:(j + 1) * coef][::-1]],
                                     h)
                worst = max(worst, abs(got / r - 1))
    # the rounding of c_0, half a unit in the last place (up to 1.1e-16 of R), and
    # the interpolation's and the other coefficients' share
    assert worst < 1.6e-16


def test_powers_of_two():
    t = _table("kExp2Table")
    assert len(t) == 64
    with mpmath.workdps(40):
        assert all(v == float(mpmath.mpf(2) ** (mpmath.mpf(j) / 64)) for j, v in enumerate(t))
