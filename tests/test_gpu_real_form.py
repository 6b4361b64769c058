"""The REAL form of the Raman and contraction kernels (couplings symmetric in (l, m): two pair fields a
slot, only Re W formed) against the general form and the oracle, for every kernel that has it: the
sparse contraction with the recurrence in the tiles, with R from transforms and with Raman off, the
serial-recurrence tall tiles, the dense form and the tensor cores; odd counts of pair fields; the
scan of the carries; a coupling that is not symmetric (which must keep the general form), and a
batch that mixes both, whose members get the bits they have alone.

Tolerance: both forms evaluate the same sums without the terms that are 0 (often to the same bits): FP32 rounding below
1e-6 of these fields, FP64 1e-13."""
import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


def _solve(mmp, prob):
    with mmp.Solver(prob) as s:
        s.propagate(prob.n_steps)
        return s.result(), s.info()


def _two_term(nt, window):
    t = np.arange(nt) * (window / nt)
    h = np.exp(-t / 0.032) * np.sin(t / 0.0122) + 0.3 * np.exp(-t / 0.1) * np.sin(t / 0.05)
    return h / (h.sum() * (window / nt))


def _prob(form, M, nnz, nt):
    if form in ("dense", "tensor"):
        p = W.dense15(seed=M, M=M, nt=nt, n_steps=3)
        return W.scale_power(p, W.phase_cap_scale(p, per_step=0.02, total=0.1))
    p = W.small_case(seed=20 + M, M=M, nt=nt, n_steps=3, raman=form != "off", nnz_target=nnz, physical_order=True,
                     peak_w=20.0)
    return p.replace(raman_response=_two_term(nt, p.time_window)) if form == "transforms" else p


CASES = [("tiles", 5, 60, 64), ("tiles", 6, 90, 1024), ("tiles", 9, 200, 2048), ("scan", 6, 90, 1024),
         ("transforms", 2, 12, 512), ("transforms", 6, 90, 2048), ("off", 6, 90, 512), ("off", 9, 200, 1024),
         ("tall", 22, 1200, 256), ("tall", 21, 1600, 2048), ("dense", 5, 0, 512), ("tensor", 6, 0, 128),
         ("tensor", 9, 0, 1024), ("tensor", 16, 0, 256)]


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("form,M,nnz,nt", CASES)
def test_matches_the_general_form(mmp, monkeypatch, form, M, nnz, nt, fp64):
    prob = _prob(form, M, nnz, nt)
    if fp64 and form in ("dense", "tensor"):  # symmetric to the last bit
        q = prob.coupling.copy()
        val = {}
        for i, e in enumerate(q):
            val.setdefault((e["p"], e["k"], min(e["l"], e["m"]), max(e["l"], e["m"])), []).append(i)
        for idx in val.values():
            q["value"][idx] = q["value"][idx[0]]
        prob = prob.replace(coupling=q)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    if form == "scan":
        monkeypatch.setenv("MMP_LOOKBACK", "0")
    out, info = _solve(mmp, prob)
    assert (info["contract_sub_block"] > 0) == (form == "tall")
    assert info["tensor_core_contraction"] == (form == "tensor" and not fp64)
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    ref, _ = _solve(mmp, prob)
    assert mo.rel_l2_per_mode(out, ref).max() < (1e-13 if fp64 else 1e-6)
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < (1e-11 if fp64 else 1e-5)


def _skewed(prob):
    """The coupling with Q_pklm and Q_pkml apart by a few percent."""
    q = prob.coupling.copy()
    up = q["l"] > q["m"]
    q["value"][up] *= 1.03
    return prob.replace(coupling=q)


def test_unsymmetric_coupling_keeps_the_general_form(mmp, monkeypatch):
    prob = _skewed(_prob("tiles", 6, 90, 1024))
    out, _ = _solve(mmp, prob)
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    ref, _ = _solve(mmp, prob)
    assert np.array_equal(out, ref)
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < 1e-5


@pytest.mark.parametrize("form,M,nnz,nt", [("tiles", 6, 90, 1024), ("transforms", 6, 90, 512), ("tall", 22, 1200, 256),
                                           ("tensor", 8, 0, 256)])
def test_mixed_batch_gives_the_bits_of_each_alone(mmp, monkeypatch, form, M, nnz, nt):
    for k, v in (("MMP_ROW_SPLIT", "0"), ("MMP_CONTRACT_TILE", "128"), ("MMP_GROUPS", "1")):
        monkeypatch.setenv(k, v)
    base = _prob(form, M, nnz, nt)
    probs = [base, _skewed(base), W.scale_power(base, 0.5)]
    alone = [_solve(mmp, p)[0] for p in probs]
    with mmp.Batch(probs) as b:
        b.propagate(base.n_steps)
        for i, ref in enumerate(alone):
            assert np.array_equal(b.result(i), ref), i


@pytest.mark.parametrize("M,nnz,nt,tile,raman", [(22, 1200, 64, 64, True), (23, 1200, 256, 64, True), (64, 1500, 128, 128, True),
                                                 (22, 1200, 256, 128, False)])
def test_tall_tiles_of_two_sub_blocks_and_up(mmp, monkeypatch, M, nnz, nt, tile, raman):
    """The FP32 tall form takes 32 samples at a time: its shortest tiles, its most rows of U, odd slot counts."""
    prob = W.small_case(seed=40 + M, M=M, nt=nt, n_steps=2, raman=raman, nnz_target=nnz, physical_order=True, peak_w=20.0)
    monkeypatch.setenv("MMP_CONTRACT_TILE", str(tile))
    out, info = _solve(mmp, prob)
    assert info["contract_sub_block"] > 0 and info["contract_tile"] == tile
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    ref, _ = _solve(mmp, prob)
    assert mo.rel_l2_per_mode(out, ref).max() < 1e-6
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < 1e-5
