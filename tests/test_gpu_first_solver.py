"""A process's first solver loads the kernels it runs, not every instantiation of the library: what loading
takes on the device is a few MB (about 30 with all of them, and 80 ms), and the other kernels still
get their shared-memory opt-in when a later solver or transform needs them."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np, torch
torch.zeros(1, device="cuda"); torch.cuda.synchronize()
import mm_propagation_b200 as mmp
from mm_propagation_b200 import capi, workloads as W
mmp.lib()
before = torch.cuda.mem_get_info()[0]
with mmp.Solver(W.small_case(seed=1, M=1, nt=64, n_steps=8, nnz_target=1)) as s:
    s.propagate(8)
    assert np.isfinite(s.result()).all()
    print((before - torch.cuda.mem_get_info()[0]) / 2**20)
# rows of 128 KB a CTA and a transform on its own
for nt, fp64 in ((16384, False), (65536, False), (8192, True), (32768, True)):
    p = W.small_case(seed=2, M=2, nt=nt, n_steps=8, window=40.0).replace(flags=capi.MMP_F_FP64 if fp64 else 0)
    for probs in ([p], [p] * 3):
        with mmp.Batch(probs) as b:
            b.propagate(8)
            assert np.isfinite(b.result(0)).all()
    x = np.random.default_rng(nt).standard_normal((2, nt)) + 0j
    assert np.abs(mmp.dft(mmp.dft(x, fp64=fp64), inverse=True, fp64=fp64) - x).max() < (1e-13 if fp64 else 1e-4)
"""


def test_only_its_own_kernels_are_loaded():
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert float(r.stdout.split()[0]) <= 16
