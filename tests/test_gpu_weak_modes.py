"""Modes far weaker than the strongest one, and dark ones: every route of the pair fields keeps a mode's
rounding relative to that mode. The coupling has entries for (p, p, r, r) and its permutations alone, so
that a dark mode stays dark and a weak one is driven by the strong ones.

Tolerance: the solve's error per mode against the FP64 oracle is at most twice that of the form that
keeps one complex pair field a slot (MMP_REAL_PAIRS=0), beyond a floor of 1e-7 in FP32 (a few
roundings of 6e-8) and 1e-13 in FP64; a dark mode is exactly 0. A pair field that shared a complex transform
with one 1e4 times as strong would carry 1e4 roundings."""
import itertools

import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu

AMPLITUDES = [1.0, 1e-8, 0.0, 0.1, 1e-4]  # of modes 0, 1, 2, ..., in turn
ROUTES = {  # M, nt, environment
    "tiles": (5, 1024, {}), "scan": (5, 1024, {"MMP_LOOKBACK": "0"}), "rows": (5, 512, {"MMP_RAMAN_FUSED": "0"}),
    "transforms": (5, 1024, {}), "two_transforms": (2, 512, {}), "off": (5, 1024, {}), "tall": (22, 256, {}),
    "dense": (5, 512, {"MMP_DENSE": "1", "MMP_TC": "0"}), "dense_transforms": (5, 512, {"MMP_DENSE": "1"}),
    "tensor": (6, 256, {"MMP_DENSE": "1"})}


def _two_term(nt, window):
    t = np.arange(nt) * (window / nt)
    h = np.exp(-t / 0.032) * np.sin(t / 0.0122) + 0.3 * np.exp(-t / 0.1) * np.sin(t / 0.05)
    return h / (h.sum() * (window / nt))


def _prob(route):
    M, nt, _ = ROUTES[route]
    p = W.small_case(seed=M, M=M, nt=nt, n_steps=20, raman=route != "off", physical_order=True, peak_w=100.0)
    rng = np.random.default_rng(M)
    entries = W.pair_prefix(M)
    for a, b in itertools.combinations_with_replacement(range(M), 2):
        v = 5e12 * np.exp(0.3 * rng.standard_normal())
        entries += [(*t, v) for t in sorted(set(itertools.permutations((a, a, b, b))))]
    p = p.replace(coupling=W.nz_array(entries))
    if route.endswith("transforms"):
        p = p.replace(raman_response=_two_term(nt, p.time_window))
    peak = np.abs(p.initial_fields).max(axis=1, keepdims=True)
    amp = np.array([AMPLITUDES[i % len(AMPLITUDES)] for i in range(M)])[:, None]
    p = p.replace(initial_fields=1e3 * p.initial_fields / peak * amp)
    return W.scale_power(p, W.phase_cap_scale(p, per_step=0.02, total=0.4))


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("route", list(ROUTES))
def test_a_weak_mode_keeps_its_own_rounding(mmp, monkeypatch, route, fp64):
    for k, v in ROUTES[route][2].items():
        monkeypatch.setenv(k, v)
    prob = _prob(route)
    ref = mo.solve(prob)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)

    def run():
        with mmp.Solver(prob) as s:
            s.propagate(prob.n_steps)
            return s.result(), s.info()

    out, info = run()
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    general, _ = run()
    assert info["raman_recurrence"] == (0 if route == "off" or route.endswith("transforms") else 1 if route == "rows" else 2)
    assert info["tensor_core_contraction"] == (route == "tensor" and not fp64)
    assert (info["contract_sub_block"] > 0) == (route == "tall")
    lit = np.abs(prob.initial_fields).max(axis=1) > 0
    assert np.all(out[~lit] == 0) and np.all(general[~lit] == 0)
    norm = np.linalg.norm(ref[lit], axis=1)
    err = np.linalg.norm(out[lit] - ref[lit], axis=1) / norm
    err_general = np.linalg.norm(general[lit] - ref[lit], axis=1) / norm
    print(route, "fp64" if fp64 else "fp32", "max err", err.max(), "general", err_general.max())
    assert np.all(err <= 2 * err_general + (1e-13 if fp64 else 1e-7)), (err, err_general)
