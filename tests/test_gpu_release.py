"""Grids of up to one block per SM, whose colour kernels let the next one in
within their subject loop (REL): segments of many sweeps, where the kernels
overlap, against single sweeps that do not, bit for bit; the probit forms against
the 8-subject step, which has no such form; and the FP64 oracle chain.
"""
from __future__ import annotations

import numpy as np
import pytest

from bsglmm_gb300 import synth

pytestmark = pytest.mark.gpu


def _chain(st, wm, model, pred, sweeps, single=False, step=0):
    import bsglmm_gb300 as bsg
    with bsg.Sampler() as s:
        ds = s.add_dataset(st.mask, st.covar, st.data, 1, wm)
        ch = s.add_chain(ds, seed=21, beta_wm=0.0 if wm is None else 0.3)
        s.set_model(ch, model)
        if wm is not None:
            s.set_wm_update(ch, True)
        if pred:
            s.set_predictive(ch, True)
        s.set_step_subjects(step)
        for _ in range(sweeps if single else 1):
            s.run(1 if single else sweeps)
        out = [s.beta(ch), s.omega(ch), s.colmeans(ch), *s.posterior(ch)[:3],
               np.array(s.beta_wm(ch))]
        return out + ([s.predictive(ch)[0]] if pred else [])


@pytest.mark.parametrize("model,N,P,first,wm,pred", [
    ("probit", 110, 2, True, False, False), ("probit", 150, 4, False, True, False),
    ("probit", 165, 5, True, True, True), ("probit", 421, 8, False, False, True),
    ("probit", 90, 1, True, False, False),
    ("t", 20, 2, True, False, False), ("t", 47, 1, True, False, False),
    ("logistic", 63, 3, False, False, True), ("t", 81, 4, True, False, False),
    ("logistic", 233, 5, True, False, False), ("t", 1100, 2, False, False, False),
])
def test_overlapped_sweeps_equal_single_ones(oracle_mod, model, N, P, first, wm, pred):
    st = synth.small_study(700 + N, shape=(17, 16, 15), N=N, P=P, S=1)
    st.covar = st.covar if first else np.ascontiguousarray(st.covar[::-1])
    w = np.random.default_rng(N).random(st.V).astype(np.float32) if wm else None
    many = _chain(st, w, model, pred, 33)
    for a, b in zip(many, _chain(st, w, model, pred, 33, single=True)):
        assert np.array_equal(a, b)
    if model == "probit":
        for a, b in zip(many, _chain(st, w, model, pred, 33, step=8)):
            assert np.array_equal(a, b)
    pb = oracle_mod.Problem(st.mask, st.covar, st.data, 1, w)
    o = pb.chain(21, 2, beta_wm=0.3 if wm else 0.0, wm_update=wm,
                 model={"logistic": 0, "probit": 1, "t": 2}[model])
    # FP32 draws of two sweeps from the oracle's
    assert np.allclose(_chain(st, w, model, pred, 2)[0], o["beta"], rtol=1e-4, atol=1e-4)
