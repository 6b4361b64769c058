"""FP64 solves whose linear phase is enormous (beta_0 z of 1e3 to 1e60 rad): exp(i theta) stays on the unit circle
for every finite phase, so the linear part conserves each mode's energy and the solve stays finite.

Tolerance: each of the 3 x 4 + 1 phase factors a sample meets is a unit vector to about 2^-52, a transform
pair a stage adds a few roundings: 1e-12 of the energy."""
import numpy as np
import pytest

from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 6])
@pytest.mark.parametrize("phase", [1e3, 1e14, 3e15, 1e16, 1e17, 1e19, 1e25, 1e60])
def test_energy_of_each_mode_is_kept(mmp, phase, order):
    p = W.small_case(seed=5, M=2, nt=256, n_steps=3, order=order, raman=False, nnz_target=2, peak_w=1.0)
    beta = p.dispersion.copy()
    beta[1, 0] = phase / p.fiber_length
    # self-phase terms alone: no energy moves between the modes; 1e-6 rad a step
    q = W.nz_array([(0, 0, 0, 0, 5e12), (1, 1, 1, 1, 5e12)])
    p = p.replace(dispersion=beta, coupling=q, flags=capi.MMP_F_FP64)
    p = W.scale_power(p, W.phase_cap_scale(p, per_step=1e-6, total=1e-5))
    with mmp.Solver(p) as s:
        s.propagate(3)
        out = s.result()
    e0 = (np.abs(p.initial_fields) ** 2).sum(axis=1)
    e1 = (np.abs(out) ** 2).sum(axis=1)
    assert np.abs(e1 / e0 - 1).max() < 1e-12
