"""A batch's z reset (one launch for its solves, or one by one where only some start over), its
status word over all solves, and new fields clearing both: each member gives the bits it gives alone."""
import numpy as np
import pytest

from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def one_shape(monkeypatch):
    for k, v in (("MMP_ROW_SPLIT", "0"), ("MMP_CONTRACT_TILE", "128"), ("MMP_GROUPS", "1")):
        monkeypatch.setenv(k, v)


@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("carry", [(0,), (0, 0, 0), (0, 1, 0), (1, 1)])
def test_second_call_starts_over_or_carries_on(mmp, carry, fp64):
    base = W.small_case(seed=7, M=3, nt=512, n_steps=6, raman=True, peak_w=20.0)
    flag = capi.MMP_F_FP64 if fp64 else 0
    probs = [W.scale_power(base, 1.0 - 0.2 * i).replace(flags=flag | (capi.MMP_F_CONTINUOUS if c else 0))
             for i, c in enumerate(carry)]
    alone = []
    for p in probs:
        with mmp.Solver(p) as s:
            s.propagate(9)
            s.propagate(6)
            alone.append(s.result())
    with mmp.Batch(probs) as b:
        b.propagate(9)
        b.propagate(6)
        for i, ref in enumerate(alone):
            assert np.array_equal(b.result(i), ref), i
        b.set_fields(0, probs[0].initial_fields)  # back at z = 0 whatever the flag
        b.propagate(9)
        b.propagate(6)
        assert np.array_equal(b.result(0), alone[0])


@pytest.mark.parametrize("where", [0, 299])
def test_one_failing_solve_of_many_is_reported_until_it_gets_new_fields(mmp, where):
    good = W.grin2(seed=2, nt=256, n_steps=400, peak_scale=0.01)
    bad = W.grin2(seed=1, nt=256, n_steps=1000, literal=True)  # diverges
    probs = [good] * 300  # more than one word a thread
    probs[where] = bad
    with mmp.Batch(probs) as b:
        with pytest.raises(mmp.MMPError) as ei:
            b.propagate(400)
        assert ei.value.code == capi.MMP_ENONFINITE
        for i in (1, 150):
            assert np.isfinite(b.result(i)).all()
        b.set_fields(where, bad.initial_fields)
        b.propagate(2)  # clean again (these fields last two steps and not four)


def test_more_solvers_alive_than_shared_words(mmp):
    """Solvers share one block of mapped words (256 of them), further ones have their own; given back when closed."""
    prob = W.small_case(seed=3, M=1, nt=64, n_steps=2, raman=False)
    bad = np.full_like(prob.initial_fields, np.nan)
    for _ in range(2):
        solvers = [mmp.Solver(prob) for _ in range(260)]
        out = []
        for s in (solvers[0], solvers[255], solvers[259]):
            with pytest.raises(mmp.MMPError):
                s.set_fields(bad)
            s.set_fields(prob.initial_fields)
            s.propagate(2)
            out.append(s.result())
        for s in solvers:
            s.close()
        assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
