"""Couplings with entries far below the largest that are not symmetric in (l, m): a mode driven by
nothing else is still right. Q_plm = delta_1, Q_pml = delta_2 on the last mode, the rest symmetric; a = delta_1 + delta_2
and b = delta_1 - delta_2 are the sum and the difference.

Tolerance: 1e-5 of the mode's norm, the bound of FP32 solves; without the b part the last mode would be 0
(a = 0) or 10% off (a = 10 b)."""
import itertools

import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi, workloads as W
from test_gpu_kernel_forms import forms
from test_gpu_real_form import _prob as symmetric_prob

pytestmark = pytest.mark.gpu

FORMS = {"tiles": (6, 1024, {}), "scan": (6, 512, {"MMP_LOOKBACK": "0"}), "off": (6, 512, {}), "tall": (22, 256, {}),
         "dense": (5, 512, {"MMP_DENSE": "1", "MMP_TC": "0"}), "tensor": (7, 256, {"MMP_DENSE": "1"})}


def _prob(form, a, b):
    M, nt, _ = FORMS[form]
    p = W.small_case(seed=M, M=M, nt=nt, n_steps=6, raman=form != "off", physical_order=True, peak_w=100.0)
    rng = np.random.default_rng(M)
    entries = W.pair_prefix(M)
    for i, j in itertools.combinations_with_replacement(range(M - 1), 2):
        v = 5e12 * np.exp(0.3 * rng.standard_normal())
        entries += [(*t, v) for t in sorted(set(itertools.permutations((i, i, j, j))))]
    top = max(e[4] for e in entries)
    entries += [(M - 1, 0, 1, 2, (a + b) / 2 * top), (M - 1, 0, 2, 1, (a - b) / 2 * top)]
    # pulses on top of one another: where only tails overlap, the drive is as small as the FP32 rounding there
    fields = np.stack([W.gaussian(nt, p.time_window, p.time_window / 20, 100.0, ph) for ph in rng.uniform(0, 6, M)])
    fields[M - 1] = 0
    p = p.replace(coupling=W.nz_array(entries), initial_fields=fields)
    return W.scale_power(p, W.phase_cap_scale(p, per_step=0.02, total=0.2))


@pytest.mark.parametrize("a,b", [(1e-11, 1e-12), (0.0, 1e-12), (0.0, 3e-16), (1e-12, 1e-12), (1e-4, 1e-10)])
@pytest.mark.parametrize("form", list(FORMS))
def test_a_mode_driven_by_small_unsymmetric_terms(mmp, monkeypatch, form, a, b):
    for k, v in FORMS[form][2].items():
        monkeypatch.setenv(k, v)
    prob = _prob(form, a, b)
    ref = mo.solve(prob)
    assert np.linalg.norm(ref[-1]) > 0
    with mmp.Solver(prob) as s:
        s.propagate(prob.n_steps)
        out, info = s.result(), s.info()
    assert info["tensor_core_contraction"] == (form == "tensor") and (info["contract_sub_block"] > 0) == (form == "tall")
    assert mo.rel_l2_per_mode(out, ref).max() < 1e-5
    assert forms(mmp, [prob])[0][1] == 0


@pytest.mark.parametrize("form", list(FORMS))
def test_rounding_left_by_a_symmetrisation_keeps_the_real_form(mmp, monkeypatch, form):
    for k, v in FORMS[form][2].items():
        monkeypatch.setenv(k, v)
    prob = _prob(form, 1e-3, 2.0 ** -56)  # the last bits of two Q next to 1e-3 of the largest
    assert forms(mmp, [prob])[0][1] == 1
    assert forms(mmp, [symmetric_prob("tensor", 9, 0, 1024)])[0][1] == 1  # 24 permutations summed in other orders
