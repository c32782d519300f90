"""The colour kernels' subject loop at the sizes where its steps change: the
ends of a ragged last outcome word (16-, 8- and 4-subject steps, the last one
partly beyond N) and the edges of a staged pass (1024 subjects, 512 for the
t/logit links), against the FP64 oracle chain on the same counters.
"""
from __future__ import annotations

import numpy as np
import pytest

from bsglmm_gb300 import synth

pytestmark = pytest.mark.gpu

# one sweep of FP32 draws from the oracle's (the bound of the other oracle
# comparisons of single sweeps)
TOL = 1e-4


def _P(N):
    """Covariates: one for the few-subject studies, whose isolated voxel would
    otherwise have a singular X'X and no neighbour to add Omega."""
    return 1 if N < 8 else 3 + N % 2


@pytest.mark.parametrize("step", [8, 16])
@pytest.mark.parametrize("N", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 31, 33, 1023, 1024, 1029])
def test_probit_sweep_matches_oracle(oracle_mod, N, step):
    import bsglmm_gb300 as bsg
    st = synth.small_study(300 + N, shape=(6, 5, 6), N=N, P=_P(N), S=1)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=7)
        s.set_step_subjects(step)
        s.run(1)
        o = oracle_mod.Problem(st.mask, st.covar, st.data, 1).chain(7, 1)
        assert np.allclose(s.beta(ch), o["beta"], rtol=TOL, atol=TOL)


@pytest.mark.parametrize("P", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("step", [8, 16])
@pytest.mark.parametrize("first", [True, False])
def test_intercept_first_or_not_matches_oracle(oracle_mod, P, step, first):
    """The form for a first design column of ones, and the general one (the
    same design with its columns in the opposite order); with the beta_WM
    update at even P."""
    import bsglmm_gb300 as bsg
    st = synth.small_study(600 + P, shape=(7, 6, 5), N=59, P=P, S=1)
    covar = st.covar if first else np.ascontiguousarray(st.covar[::-1])
    assert (covar[0] == 1).all() == first
    wm = np.random.default_rng(P).random(st.V).astype(np.float32) if P % 2 == 0 else None
    with bsg.Sampler() as s:
        ds = s.add_dataset(st.mask, covar, st.data, 1, wm)
        ch = s.add_chain(ds, seed=13, beta_wm=0.0 if wm is None else 0.3)
        if wm is not None:
            s.set_wm_update(ch, True)
        s.set_step_subjects(step)
        s.run(1)
        pb = oracle_mod.Problem(st.mask, covar, st.data, 1, wm)
        o = pb.chain(13, 1, beta_wm=0.0 if wm is None else 0.3, wm_update=wm is not None)
        assert np.allclose(s.beta(ch), o["beta"], rtol=TOL, atol=TOL)


@pytest.mark.parametrize("N", [1, 30, 32, 35, 511, 512, 513, 1030])
def test_t_sweep_matches_oracle(oracle_mod, N):
    import bsglmm_gb300 as bsg
    st = synth.small_study(400 + N, shape=(6, 5, 6), N=N, P=_P(N), S=1)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=9)
        s.set_model(ch, "t")
        s.run(1)
        o = oracle_mod.Problem(st.mask, st.covar, st.data, 1).chain(9, 1, model=2)
        assert np.allclose(s.beta(ch), o["beta"], rtol=TOL, atol=TOL)


@pytest.mark.parametrize("N", [1, 2, 3, 5, 6, 31, 33, 511, 512, 513])
def test_fp64_sweep_matches_oracle(oracle_mod, N):
    """FP64 chains on four lanes per voxel: quads of subjects, a short last
    pair, the 512-subject pass."""
    import bsglmm_gb300 as bsg
    st = synth.small_study(500 + N, shape=(6, 5, 6), N=N, P=_P(N), S=1)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(st.mask, st.covar, st.data, 1), seed=11)
        s.set_precision(ch, 64)
        s.run(1)
        o = oracle_mod.Problem(st.mask, st.covar, st.data, 1).chain(11, 1)
        # FP64 on both sides: rounding, with room for the draw's conditioning
        assert np.allclose(s.beta64(ch), o["beta"], rtol=1e-11, atol=1e-11)


def test_fp64_one_lane_matches_oracle(oracle_mod):
    """The same on one lane per voxel (38,912 voxels a colour and more)."""
    import bsglmm_gb300 as bsg
    rng = np.random.default_rng(77)
    mask = np.ones((44, 43, 42), np.uint8)  # 39,732 voxels of each colour
    N, V = 7, int(mask.sum())
    covar = np.stack([np.ones(N), rng.standard_normal(N)]).astype(np.float32)
    data = (rng.random((N, V)) < 0.2).astype(np.uint8)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(mask, covar, data, 1), seed=12)
        s.set_precision(ch, 64)
        s.run(1)
        o = oracle_mod.Problem(mask, covar, data, 1).chain(12, 1)
        assert np.allclose(s.beta64(ch), o["beta"], rtol=1e-11, atol=1e-11)
