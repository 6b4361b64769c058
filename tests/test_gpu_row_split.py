"""The row split of solves that are not tuned, where the rows just fill the chip: clusters lie within groups
of SMs, so fewer of them are resident than SMs / CTAs suggests, and a split whose clusters
need a second wave is slower than rows left whole (26-30 us a k_nu launch against 20 before 16, 17 and
18 rows of 8 CTAs and 34 to 37 of 4 were counted as two waves).

Bound: k_nu no more than a tenth slower than with whole rows (repeated minima differ by about 3%)."""
import pytest

from mm_propagation_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [15, 16, 17, 18, 33, 34, 36, 37])
def test_a_split_row_is_not_slower_than_a_whole_one(mmp, monkeypatch, M):
    p = W.small_case(seed=M, M=M, nt=8192, n_steps=8, window=20.0, physical_order=True, peak_w=1.0, nnz_target=300)

    def k_nu():
        with mmp.Batch([p]) as b:
            b.propagate(8)
            return min(b.profile(4)["nu"]["ms_per_launch"] for _ in range(6)), b.info(0)["cluster_ctas"]

    split, ctas = k_nu()
    monkeypatch.setenv("MMP_ROW_SPLIT", "0")
    whole, one = k_nu()
    assert one == 1 and ctas > 1
    assert split <= 1.1 * whole
