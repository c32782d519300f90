"""Block sizes per launch group (the default), one for all groups, and back:
which the plan uses, that the chains do not depend on it, and that the autotuner
leaves the choice per group open.
"""
from __future__ import annotations

import numpy as np
import pytest

from bsglmm_gb300 import synth

pytestmark = pytest.mark.gpu


def _cube(shape, N, P, seed):
    rng = np.random.default_rng(seed)
    X, Y, Z = shape
    mask = (rng.random((Z, Y, X)) < 0.9).astype(np.uint8)
    covar = np.ones((P, N), np.float32)
    covar[1:] = rng.standard_normal((P - 1, N)).astype(np.float32)
    return mask, covar, (rng.random((N, int(mask.sum()))) < 0.2).astype(np.uint8)


@pytest.mark.parametrize("N,P,wm,model,bits,want", [
    (170, 3, False, "probit", 32, 128), (170, 5, True, "probit", 32, 128),
    (20, 3, False, "probit", 32, 256), (40, 3, False, "logistic", 32, 128),
    (40, 6, False, "t", 32, 128), (33, 8, False, "logistic", 32, 128),
    (20, 3, False, "probit", 64, 64),
])
def test_default_block_size_of_a_small_grid(N, P, wm, model, bits, want):
    import bsglmm_gb300 as bsg
    mask, covar, data = _cube((18, 17, 16), N, P, 40 + P)
    with bsg.Sampler() as s:
        w = np.full(int(mask.sum()), 0.5, np.float32) if wm else None
        ch = s.add_chain(s.add_dataset(mask, covar, data, 1, w), seed=5)
        s.set_model(ch, model)
        s.set_precision(ch, bits)
        if wm:
            s.set_wm_update(ch, True)
        assert s.block_threads(ch) == want


def test_sizes_per_group_come_back():
    import bsglmm_gb300 as bsg
    a, b = _cube((18, 17, 16), 170, 3, 1), _cube((13, 12, 11), 21, 4, 2)
    out = []
    for how in ("default", "set and back", "autotuned and back"):
        with bsg.Sampler() as s:
            ids = [s.add_chain(s.add_dataset(*x, 1), seed=5) for x in (a, b)]
            if how == "set and back":
                s.set_tuning(0, 64)
                assert [s.block_threads(c) for c in ids] == [64, 64]
            elif how == "autotuned and back":
                lpv, thr = s.autotune(2)
                assert (lpv, thr) == s.tuning()
                s.set_tensor_xz(False)
                s.set_step_subjects(0)
            if how != "default":
                s.set_tuning(1, -1)
            assert [s.block_threads(c) for c in ids] == [128, 256]
            assert s.tuning() == (1, 256)
            s.set_tuning(0, 0)  # keeps it
            assert [s.block_threads(c) for c in ids] == [128, 256]
            s.run(5)
            out.append([x for c in ids for x in (s.beta(c), s.omega(c))])
            with pytest.raises(bsg.BsgError):
                s.set_tuning(0, -2)
            with pytest.raises(bsg.BsgError):
                s.block_threads(2)
    for o in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o, out[0]))


@pytest.mark.parametrize("first", [True, False])
def test_tensor_xz_switch_on_a_running_context(first):
    """Switched after the plan was built, the tensor-core X'Z is what runs:
    the same chain as with the plan rebuilt (another block size, same results)."""
    import bsglmm_gb300 as bsg
    st = synth.small_study(9, shape=(12, 11, 10), N=70, P=4, S=1)
    covar = st.covar if first else np.ascontiguousarray(st.covar[::-1])
    out = []
    for rebuild in (False, True):
        with bsg.Sampler() as s:
            ch = s.add_chain(s.add_dataset(st.mask, covar, st.data, 1), seed=5)
            s.run(1)
            assert s.step_subjects() == 16
            s.set_tensor_xz(True)
            if rebuild:
                s.set_tuning(1, 64)
            s.run(1)
            assert s.step_subjects() == 8
            out.append(s.beta(ch))
    assert np.array_equal(out[0], out[1])
