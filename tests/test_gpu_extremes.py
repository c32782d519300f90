"""Inputs at the edge of what the kernels' arithmetic takes, against the FP64
oracle chain on the same counters: far tails, designs beyond a float's range.
"""
from __future__ import annotations

import numpy as np
import pytest

from bsglmm_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [33, 52, 64, 77])
def test_tensor_xz_far_tail_in_a_ragged_last_word(oracle_mod, N):
    """beta_WM WM = 15: beyond N the tensor-core form's last word has
    a = 15, where the inversion is not finite; x = 0 there, so the sweep is
    that of the other subjects."""
    import bsglmm_gb300 as bsg
    st = synth.small_study(41, shape=(9, 8, 7), N=N, P=4, S=1)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=9, beta_wm=15.0)
        s.set_tensor_xz(True)
        s.run(1)
        b = s.beta(ch)
    o = oracle_mod.Problem(st.mask, st.covar, st.data, 1).chain(9, 1, beta_wm=15.0)
    # the split product's 2^-16 of |z - beta_WM WM| < 17, twice over
    assert np.allclose(b, o["beta"], rtol=1e-4, atol=2 * 17 * 2.0 ** -16)


@pytest.mark.parametrize("bwm", [-36.0, -37.5, -200.0, -1e6, -1e14, -1e20, -1e30])
def test_fp64_far_from_the_outcome(oracle_mod, bwm):
    """FP64 chains with a mean far beyond the table of the Mills ratio, on
    the outcome's own side (|a| up to 1e30; the far side is the tail
    sampler's): finite, and the oracle's sweep."""
    import bsglmm_gb300 as bsg
    st = synth.small_study(42, shape=(9, 8, 7), N=37, P=3, S=1)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=9, beta_wm=bwm)
        s.set_precision(ch, 64)
        s.run(1)
        b = s.beta64(ch)
    o = oracle_mod.Problem(st.mask, st.covar, st.data, 1).chain(9, 1, beta_wm=float(
        np.float32(bwm)))
    # FP64 on both sides: sums of N terms of up to |beta_WM|
    assert np.allclose(b, o["beta"], rtol=1e-11, atol=1e-11 * (1.0 + abs(bwm)))


@pytest.mark.parametrize("model,P", [("probit", 2), ("probit", 6), ("t", 2), ("t", 7),
                                     ("logistic", 3)])
def test_squares_beyond_a_float(model, P):
    """A first column of about 2e19: its sum of squares is infinite in FP32 and
    its coefficient's conditional a spike at 0, as the division by its pivot
    gives; the others' draws go on."""
    import bsglmm_gb300 as bsg
    rng = np.random.default_rng(4)
    N, mask = 40, np.ones((6, 6, 6), np.uint8)
    covar = rng.standard_normal((P, N)).astype(np.float32)
    covar[0] *= 2e19
    covar[-1] = 1
    data = (rng.random((N, 216)) < 0.3).astype(np.uint8)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(mask, covar, data, 1), seed=9)
        s.set_model(ch, model)
        s.run(1)
        b = s.beta(ch)
        s.run(3)
        assert np.isfinite(s.beta(ch)).all() and not s.beta(ch)[0].any()
    assert not b[0].any()
    # bounded regression coefficients of a 0/1 outcome on unit-scale columns
    assert np.abs(b[1:]).max() < 5 and (b[1:] != 0).any(axis=1).all()
