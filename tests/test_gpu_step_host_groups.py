"""bsg_step_host on contexts of several launch groups (chains of different P, links
and precision): steps of one to four sweeps equal bsg_set_omega, bsg_run and the
getters, bit for bit, for every chain of the context.
"""
from __future__ import annotations

import numpy as np
import pytest

from bsglmm_gb300 import synth

pytestmark = pytest.mark.gpu


def _context(groups):
    import bsglmm_gb300 as bsg
    s = bsg.Sampler()
    for k, (P, model, bits, pred) in enumerate(groups):
        st = synth.small_study(60 + k, shape=(9, 8, 7), N=30 + 9 * k, P=P, S=1)
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=70 + k)
        s.set_model(ch, model)
        s.set_precision(ch, bits)
        s.set_predictive(ch, pred)
    return s


@pytest.mark.parametrize("groups", [
    [(3, "probit", 32, True)],
    [(2, "probit", 32, False), (4, "probit", 32, False)],
    [(3, "probit", 32, True), (3, "t", 32, False), (2, "probit", 64, False),
     (5, "logistic", 32, True), (6, "probit", 32, False)],
])
def test_steps_equal_separate_calls(groups):
    with _context(groups) as a, _context(groups) as b:
        n_ch = len(groups)
        for k in range(8):
            ch, n = k % n_ch, 1 + k % 4
            om = np.eye(groups[ch][0]) * (1.5 + k) + 0.1 if k % 3 == 0 else None
            o1, c1 = a.step_host(ch, om, n)
            if om is not None:
                b.set_omega(ch, om)
            b.run(n)
            assert np.array_equal(o1, b.omega(ch)) and np.array_equal(c1, b.colmeans(ch))
        for ch in range(n_ch):
            assert np.array_equal(a.beta64(ch), b.beta64(ch))
            assert np.array_equal(a.omega(ch), b.omega(ch))
            for x, y in zip(a.posterior(ch)[:3], b.posterior(ch)[:3]):
                assert np.array_equal(x, y)
            if groups[ch][3]:
                assert np.array_equal(a.predictive(ch)[0], b.predictive(ch)[0])
