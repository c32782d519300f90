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
