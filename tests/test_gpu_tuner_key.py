"""The autotuner's choice is cached per shape: batches that run other kernels are other shapes, whatever was
created before them in the process."""
import itertools

import numpy as np
import pytest

from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


def _two_term(nt, window):
    t = np.arange(nt) * (window / nt)
    h = np.exp(-t / 0.032) * np.sin(t / 0.0122) + 0.3 * np.exp(-t / 0.1) * np.sin(t / 0.05)
    return h / (h.sum() * (window / nt))


def test_other_kernels_are_other_shapes(mmp, monkeypatch):
    lib = capi.load()

    def tuned(prob):
        """Whether creating a batch of three timed anything."""
        before = lib.mmp_debug_tuned_shapes()
        with mmp.Batch([prob] * 3) as b:
            assert b.info(0)["autotuned"] == 1
        return lib.mmp_debug_tuned_shapes() - before

    M = 4
    damped = W.small_case(seed=3, M=M, nt=512, n_steps=4, physical_order=True)
    few = W.pair_prefix(M)
    for a, b in itertools.combinations_with_replacement(range(M), 2):
        few += [(*t, 5e12) for t in sorted(set(itertools.permutations((a, a, b, b))))]
    damped = damped.replace(coupling=W.nz_array(few))
    measured = damped.replace(raman_response=_two_term(512, damped.time_window))
    many = damped.replace(coupling=W.nz_array(W.pair_prefix(M) + [(*t, 5e12) for t in itertools.product(range(M), repeat=4)]))
    monkeypatch.setenv("MMP_DENSE", "0")
    assert [tuned(p) for p in (damped, damped, measured, measured, damped, many, many)] == [1, 0, 1, 0, 0, 1, 0]
    monkeypatch.setenv("MMP_LOOKBACK", "0")
    assert [tuned(p) for p in (damped, damped)] == [1, 0]
    monkeypatch.setenv("MMP_RAMAN_FUSED", "0")
    assert [tuned(p) for p in (damped, damped)] == [1, 0]
