"""Blocks of 64, 128 and 256 threads: the sums over the voxels combine in one
order, so chains agree bit for bit.  Both forms of the last block's sums (up
to 64 tiles of 256 voxels, and beyond), ragged last blocks, kept sums, the
beta_WM update and several chains.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _study(shape, N, P, seed):
    rng = np.random.default_rng(seed)
    X, Y, Z = shape
    mask = (rng.random((Z, Y, X)) < 0.9).astype(np.uint8)
    covar = np.ones((P, N), np.float32)
    covar[1:] = rng.standard_normal((P - 1, N)).astype(np.float32)
    data = (rng.random((N, int(mask.sum()))) < 0.2).astype(np.uint8)
    return mask, covar, data


def _run(study, threads, wm, chains=2, sweeps=3, model=None):
    import bsglmm_gb300 as bsg
    mask, covar, data = study
    w = np.random.default_rng(3).random(int(mask.sum())).astype(np.float32)
    out = []
    with bsg.Sampler() as s:
        ds = s.add_dataset(mask, covar, data, 1, w if wm else None)
        ids = [s.add_chain(ds, seed=5 + c, beta_wm=0.2 if wm else 0.0) for c in range(chains)]
        for c in ids:
            if wm:
                s.set_wm_update(c, True)
            if model:
                s.set_model(c, model)
        if threads:
            s.set_tuning(1, threads)
        s.run(sweeps)
        for c in ids:
            out += [s.beta(c), s.omega(c), s.colmeans(c), *s.posterior(c)[:3], s.beta_wm(c)]
    return out


@pytest.mark.parametrize("shape,N,P,wm", [
    ((7, 6, 5), 20, 3, False),      # one partial block
    ((21, 20, 19), 37, 5, True),    # 15 tiles
    ((34, 33, 33), 18, 2, False),   # 64 or 65 tiles
    ((40, 41, 42), 21, 8, False),   # over 64 tiles
    ((40, 41, 42), 21, 4, True),
])
def test_block_sizes_agree_bit_for_bit(shape, N, P, wm):
    study = _study(shape, N, P, 11 + P)
    want = _run(study, 256, wm)
    for threads in (64, 128):
        for a, b in zip(_run(study, threads, wm), want):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("N,P,wm,model", [
    (170, 3, False, None), (170, 5, True, None),
    (40, 3, False, "logistic"), (40, 6, False, "t"), (33, 8, False, "logistic"),
])
def test_block_size_of_a_small_grid_gives_the_same_chain(N, P, wm, model):
    """Few voxels and many subjects: blocks of 128 by default (above P = 5 the
    t/logit kernel's form for them), against 256 and 64 set."""
    study = _study((18, 17, 16), N, P, 40 + P)
    want = _run(study, 0, wm, model=model)
    for threads in (64, 256):
        for a, b in zip(_run(study, threads, wm, model=model), want):
            assert np.array_equal(a, b)
