"""Several threads waiting on one batch: each synchronize reports the batch's status."""
import threading

import pytest

from mm_propagation_b200 import capi, workloads as W

pytestmark = pytest.mark.gpu


def test_every_thread_that_waits_sees_the_failure(mmp):
    bad = W.grin2(seed=1, nt=256, n_steps=1000, literal=True)  # diverges
    with mmp.Batch([bad, bad]) as b:
        with pytest.raises(mmp.MMPError):
            b.propagate(400)
        seen = []

        def wait():
            for _ in range(2000):
                try:
                    b.synchronize()
                    seen.append(capi.MMP_OK)
                except mmp.MMPError as e:
                    seen.append(e.code)

        threads = [threading.Thread(target=wait) for _ in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert len(seen) == 12000 and set(seen) == {capi.MMP_ENONFINITE}
