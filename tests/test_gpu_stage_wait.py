"""The bounded waits inside k_contract_tc, between the builder warps and the thread that issues the
matrix instructions: given 0 polls (MMP_STAGE_WAIT_POLLS) they give up at once, warp by warp; the
CTA drains its copies, frees its tensor memory and reports MMP_ETIMEOUT, and the device stays usable."""
import numpy as np
import pytest

import mmp_oracle as mo
from mm_propagation_b200 import capi
from test_gpu_real_form import _prob, _skewed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [True, False])
@pytest.mark.parametrize("M,nt", [(6, 128), (9, 1024), (16, 256)])  # 3, 6 and 17 chunks of four stages
def test_stage_waits_run_out_and_report_timeout(mmp, monkeypatch, M, nt, real):
    prob = _prob("tensor", M, 0, nt)
    if not real:
        prob = _skewed(prob)
    monkeypatch.setenv("MMP_STAGE_WAIT_POLLS", "0")
    s = mmp.Solver(prob)
    monkeypatch.delenv("MMP_STAGE_WAIT_POLLS")
    with s:
        assert s.info()["tensor_core_contraction"] == 1
        for _ in range(2):
            with pytest.raises(mmp.MMPError) as ei:
                s.propagate(prob.n_steps)
            assert ei.value.code == capi.MMP_ETIMEOUT
            s.set_fields(prob.initial_fields)  # clears the status
    with mmp.Solver(prob) as s:
        s.propagate(prob.n_steps)
        out = s.result()
    assert np.isfinite(out).all() and mo.rel_l2_per_mode(out, mo.solve(prob)).max() < 1e-5
