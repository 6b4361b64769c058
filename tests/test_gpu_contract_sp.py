"""The sparse contraction of tiles of 64 to 256 samples (k_contract_sp): every tile size, rows of one
tile, one mode, more pair fields than warps and fewer, the three Raman routes and Raman off, both
precisions, against the term loop it replaces (k_contract, MMP_CONTRACT_SP=0) and the oracle; and
in a batch with dense solves, whose kernel runs beside it.

Tolerance: both evaluate the same sums of at most a few hundred products in another order: FP32
rounding (6e-8 each, relative L2 well below 1e-6 after a few steps at these powers) and FP64."""
import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


def _solve(mmp, prob):
    with mmp.Solver(prob) as s:
        s.propagate(prob.n_steps)
        return s.result(), s.info()


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("raman", ["tiles", "rows", "off"])
@pytest.mark.parametrize("M,nnz,nt,tile", [(1, 1, 64, 64), (1, 1, 2048, 256), (2, 16, 128, 128), (3, 14, 512, 64),
                                           (4, 30, 1024, 128), (6, 60, 4096, 256), (9, 160, 512, 256)])
def test_matches_the_term_loop(mmp, monkeypatch, M, nnz, nt, tile, raman, fp64):
    prob = W.small_case(seed=40 + M, M=M, nt=nt, n_steps=3, order=6, raman=raman != "off", nnz_target=nnz)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    monkeypatch.setenv("MMP_CONTRACT_TILE", str(tile))
    if raman == "rows":
        monkeypatch.setenv("MMP_RAMAN_FUSED", "0")
    out, info = _solve(mmp, prob)
    assert info["dense_contraction"] == 0 and info["contract_tile"] >= 64
    monkeypatch.setenv("MMP_CONTRACT_SP", "0")
    ref, _ = _solve(mmp, prob)
    assert mo.rel_l2_per_mode(out, ref).max() < (1e-13 if fp64 else 1e-6)
    assert mo.rel_l2_per_mode(out, mo.solve(prob)).max() < (1e-11 if fp64 else 1e-5)


@pytest.mark.parametrize("fp64", [True, False])
def test_mixed_with_dense_solves(mmp, monkeypatch, fp64):
    # a batch of two sparse solves and a dense one: each gets the kernel it gets alone
    monkeypatch.setenv("MMP_CONTRACT_TILE", "128")
    monkeypatch.setenv("MMP_TC", "0")
    dense = W.dense15(seed=7, M=5, nt=512, n_steps=3)
    dense = W.scale_power(dense, W.phase_cap_scale(dense, per_step=0.02, total=0.1))
    probs = [W.small_case(seed=60, M=3, nt=512, n_steps=3), dense, W.small_case(seed=61, M=5, nt=512, n_steps=3)]
    probs = [p.replace(flags=capi.MMP_F_FP64 if fp64 else 0) for p in probs]
    alone = [_solve(mmp, p) for p in probs]
    assert [i["dense_contraction"] for _, i in alone] == [0, 1, 0]
    with mmp.Batch(probs) as b:
        b.propagate(3)
        for i, (ref, _) in enumerate(alone):
            assert b.info(i)["dense_contraction"] == alone[i][1]["dense_contraction"]
            assert mo.rel_l2_per_mode(b.result(i), ref).max() < (1e-13 if fp64 else 1e-6)
