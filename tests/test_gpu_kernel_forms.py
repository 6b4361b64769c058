"""Which kernels a solve runs (mmp_debug_batch_form): the cases of test_gpu_real_form and test_gpu_contract_sp
compare a form with the one it replaces, which proves nothing of a form that is not taken."""
import ctypes as C

import pytest

from mm_propagation_b200 import capi, workloads as W
from test_gpu_real_form import CASES, _prob, _skewed

pytestmark = pytest.mark.gpu


def forms(mmp, probs, smem=False):
    """(merged terms, real pair fields[, shared memory of the contraction]) of each member."""
    lib = capi.load()
    with mmp.Batch(probs) as b:
        out = []
        for i in range(len(probs)):
            v = [C.c_uint32(9) for _ in range(3)]
            assert lib.mmp_debug_batch_form(b._ptr, i, *(C.byref(x) for x in v)) == capi.MMP_OK
            out.append(tuple(x.value for x in v[:3 if smem else 2]))
        assert lib.mmp_debug_batch_form(b._ptr, len(probs), None, None, None) == capi.MMP_EINVAL
        return out


def symmetric(prob):
    """Q_pklm and Q_pkml equal to the last bit."""
    q = prob.coupling.copy()
    first = {}
    for i, e in enumerate(q):
        q["value"][i] = first.setdefault((e["p"], e["k"], min(e["l"], e["m"]), max(e["l"], e["m"])), q["value"][i])
    return prob.replace(coupling=q)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("form,M,nnz,nt", [c for c in CASES if c[0] != "transforms"])
def test_symmetric_couplings_take_the_real_form(mmp, monkeypatch, form, M, nnz, nt, fp64):
    prob = symmetric(_prob(form, M, nnz, nt)).replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    if form == "scan":
        monkeypatch.setenv("MMP_LOOKBACK", "0")
    sparse = int(form in ("tiles", "scan", "off"))
    # 152 rows of 64 FP64 samples take more than the 100 KB of a tile: the term loop on shorter ones
    assert forms(mmp, [prob]) == [(sparse, int(not (fp64 and M == 16)))]
    assert forms(mmp, [_skewed(prob)]) == [(sparse, 0)]
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    assert forms(mmp, [prob])[0][1] == 0


@pytest.mark.parametrize("form,M,nnz,nt", [("tiles", 6, 90, 1024), ("tall", 22, 1200, 256), ("tensor", 8, 0, 256)])
def test_a_batch_holds_both_forms(mmp, form, M, nnz, nt):
    base = _prob(form, M, nnz, nt)
    assert [r for _, r in forms(mmp, [base, _skewed(base), W.scale_power(base, 0.5)])] == [1, 0, 1]


@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("M,nnz,nt,tile", [(1, 1, 64, 64), (2, 16, 128, 128), (6, 60, 4096, 256), (9, 160, 512, 256)])
def test_sparse_tiles_read_merged_terms(mmp, monkeypatch, M, nnz, nt, tile, fp64):
    prob = W.small_case(seed=40 + M, M=M, nt=nt, n_steps=3, order=6, nnz_target=nnz)
    prob = prob.replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    monkeypatch.setenv("MMP_CONTRACT_TILE", str(tile))
    assert forms(mmp, [prob])[0][0] == 1
    monkeypatch.setenv("MMP_CONTRACT_SP", "0")
    assert forms(mmp, [prob])[0][0] == 0


@pytest.mark.parametrize("fp64", [True, False])
def test_sparse_neighbours_cost_a_dense_solve_nothing(mmp, monkeypatch, fp64):
    """Beside solves whose contraction reads merged terms, the dense kernel holds no terms in shared memory."""
    monkeypatch.setenv("MMP_CONTRACT_TILE", "64")
    monkeypatch.setenv("MMP_TC", "0")
    monkeypatch.setenv("MMP_REAL_PAIRS", "0")
    dense = _prob("dense", 6, 0, 512)
    sparse = W.small_case(seed=60, M=3, nt=512, n_steps=3)
    dense, sparse = (p.replace(flags=capi.MMP_F_FP64 if fp64 else 0) for p in (dense, sparse))
    alone = forms(mmp, [dense], smem=True)[0]
    mixed = forms(mmp, [dense, sparse], smem=True)
    assert alone[0] == mixed[0][0] == 0 and mixed[1][0] == 1
    assert mixed[0][2] == alone[2]
