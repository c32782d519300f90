"""The predictive pass where its blocks change: subjects in one full block (256), in
two or three blocks that share the outcome words out, a last block with spare
warps; and two chains of unlike N in one launch.  Mpredict, ED and DE against the
oracle on the same coefficients.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _study(seed, N, shape=(7, 6, 5), S=2, P=4):
    rng = np.random.default_rng(seed)
    X, Y, Z = shape
    mask = (rng.random((Z, Y, X)) < 0.7).astype(np.uint8)
    grp = rng.integers(0, S, N)
    covar = rng.standard_normal((P, N)).astype(np.float32)
    for g in range(S):
        covar[g] = grp == g
    data = (rng.random((N, int(mask.sum()))) < 0.3).astype(np.uint8)
    return mask, covar, data


@pytest.mark.parametrize("N", [31, 32, 33, 255, 256, 257, 403, 513])
def test_predict_and_dic_over_blocks_of_subjects(oracle_mod, N):
    import bsglmm_gb300 as bsg
    mask, covar, data = _study(N, N)
    pb = oracle_mod.Problem(mask, covar, data, 2)
    sub = np.argmax(covar[:2] != 0, axis=0)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(mask, covar, data, 2), seed=77, burnin=0)
        s.set_predictive(ch, True)
        ed = 0.0
        for sweep in range(3):
            s.run(1)
            want = pb.predict(s.beta(ch).astype(np.float64))
            # FP32 log likelihoods of V voxels per subject, as in the other oracle tests
            assert np.allclose(s.predict(ch), want, rtol=1e-5, atol=1e-3)
            if sweep > 0:
                ed += want[np.arange(N), sub].sum()
        assert s.predictive(ch)[1] == pytest.approx(ed, rel=1e-5)
        assert s.dic(ch)["DE"] == pytest.approx(pb.dic_de(s.posterior(ch)[0]), rel=1e-5)


def test_chains_of_unlike_subjects_share_a_launch():
    """30, 403 and 257 subjects, same P and S: one launch, blocks sized for 403."""
    import bsglmm_gb300 as bsg
    studies = [_study(5, 30), _study(6, 403, shape=(17, 16, 15)), _study(7, 257)]

    def read(s, c):
        return [s.predict(c), *s.predictive(c), s.dic(c)["DE"], s.beta(c)]

    with bsg.Sampler() as s:
        ids = [s.add_chain(s.add_dataset(*x, 2), seed=9) for x in studies]
        base = s.launches_per_sweep()
        for c in ids:
            s.set_predictive(c, True)
        assert s.launches_per_sweep() == base + 2
        s.run(4)
        together = [read(s, c) for c in ids]
    for k, x in enumerate(studies):
        with bsg.Sampler() as s:
            tiny = s.add_dataset(*_study(1, 20, shape=(4, 4, 4)), 2)
            for _ in range(k):  # the chain's id is part of its variates
                s.add_chain(tiny, seed=1)
            c = s.add_chain(s.add_dataset(*x, 2), seed=9)
            s.set_predictive(c, True)
            s.run(4)
            for a, b in zip(together[k], read(s, c)):
                assert np.array_equal(a, b)
