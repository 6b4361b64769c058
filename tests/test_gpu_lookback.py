"""The states entering the contraction tiles: summed by the tiles themselves from the aggregates
before them (tile_carry) against the scan of k_raman_carry, for every contraction form, rows
shorter than the memory of the recurrence, tiles of 64 to 256 samples, and rows too long for a
slow response (which keep the scan).

Tolerance: a tile looks back until |lambda|^n < 1e-11 (FP32) or 1e-20 (FP64), so the two routes
differ by rounding: of one FP32 state (6e-8) carried into a nonlinear phase well below a
radian, or of FP64 sums (a few 1e-16); 1e-6 and 1e-13 leave an order of magnitude."""
import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu

def _solve(mmp, prob):
    with mmp.Solver(prob) as s:
        l0 = mmp.lib().mmp_kernel_launch_count()
        s.propagate(prob.n_steps)
        n = mmp.lib().mmp_kernel_launch_count() - l0
        return s.result(), s.info(), n


def _prob(form, nt, window):
    if form == "dense":
        p = W.dense15(seed=5, M=6, nt=nt, n_steps=3)
        return W.scale_power(p, W.phase_cap_scale(p, per_step=0.02, total=0.1))
    if form == "tall":
        return W.small_case(seed=12, M=22, nt=nt, n_steps=3, nnz_target=1200, physical_order=True, peak_w=20.0,
                            window=window)
    return W.small_case(seed=11, M=3, nt=nt, n_steps=4, window=window)


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("form,env,nt,window", [
    ("terms", {}, 64, 10.0), ("terms", {}, 512, 10.0), ("terms", {}, 2048, 1.0),
    ("terms", {"MMP_CONTRACT_TILE": "64"}, 1024, 4.0), ("terms", {"MMP_CONTRACT_TILE": "128"}, 16384, 20.0),
    ("dense", {}, 128, 20.0), ("dense", {}, 2048, 20.0), ("tall", {}, 256, 10.0), ("tall", {}, 4096, 10.0),
    ("tall", {"MMP_CONTRACT_SR": "0"}, 1024, 10.0)])
def test_lookback_equals_the_scan(mmp, monkeypatch, form, env, nt, window, fp64):
    prob = _prob(form, nt, window)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    out, info, n = _solve(mmp, prob)
    assert info["raman_recurrence"] == 2
    monkeypatch.setenv("MMP_LOOKBACK", "0")
    ref, _, n0 = _solve(mmp, prob)
    assert n0 == n + prob.n_steps * prob.n_stages  # one launch a stage less
    assert mo.rel_l2_per_mode(out, ref).max() < (1e-13 if fp64 else 1e-6)
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < (1e-11 if fp64 else 1e-5)


def test_short_rows_look_around_the_period(mmp):
    # 16 tiles of 256 samples: a response ten times slower than the usual one is still remembered
    # after a whole row, whose tiles are then all summed (with the period's closing factor)
    prob = W.small_case(seed=11, M=3, nt=4096, n_steps=4, window=1.0)
    t = np.arange(4096) * (1.0 / 4096)
    h = np.exp(-t / 0.32) * np.sin(t / 0.0122)
    slow = prob.replace(raman_response=h / (h.sum() / 4096))
    counts = []
    for p in (prob, slow):
        out, info, n = _solve(mmp, p)
        assert info["raman_recurrence"] == 2
        assert mo.rel_l2_per_mode(out, mo.solve(p)).max() < 1e-5
        counts.append(n)
    assert counts[0] == counts[1]


def test_long_rows_of_a_slow_response_scan(mmp, monkeypatch):
    monkeypatch.setenv("MMP_CONTRACT_TILE", "64")
    prob = W.small_case(seed=11, M=3, nt=4096, n_steps=4, window=1.0)
    out, info, n = _solve(mmp, prob)  # 51 tiles to 1e-11: the scan
    monkeypatch.setenv("MMP_LOOKBACK", "0")
    ref, _, n0 = _solve(mmp, prob)
    assert n0 == n and np.array_equal(out, ref)
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < 1e-5
