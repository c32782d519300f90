"""FP64 chains on both sides of the line between one and four lanes per voxel, at
studies where it runs through the subjects, against the FP64 oracle chain.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,N,P", [
    ((30, 30, 28), 29, 2), ((30, 30, 28), 30, 2),   # 12,600 voxels a colour
    ((30, 30, 28), 74, 5), ((30, 30, 28), 75, 5),
    ((33, 34, 33), 173, 2), ((33, 34, 33), 174, 2),  # 18,513
    ((14, 13, 12), 2, 1), ((14, 13, 12), 9, 8),      # 1,092: four from the first subjects
])
def test_fp64_sweeps_match_oracle(oracle_mod, shape, N, P):
    import bsglmm_gb300 as bsg
    rng = np.random.default_rng(N + P)
    X, Y, Z = shape
    mask = np.ones((Z, Y, X), np.uint8)
    covar = rng.standard_normal((P, N)).astype(np.float32)
    covar[0] = 1
    data = (rng.random((N, mask.size)) < 0.2).astype(np.uint8)
    with bsg.Sampler() as s:
        ch = s.add_chain(s.add_dataset(mask, covar, data, 1), seed=12)
        s.set_precision(ch, 64)
        s.run(2)
        o = oracle_mod.Problem(mask, covar, data, 1).chain(12, 2)
        # FP64 on both sides: rounding, with room for the draw's conditioning
        assert np.allclose(s.beta64(ch), o["beta"], rtol=1e-11, atol=1e-11)
