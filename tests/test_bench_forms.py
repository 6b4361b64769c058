"""The flop models of the forms that run (bench.stage_flops with merged terms and the real form,
bench.tc_mma_flops, bench.tc_useful_flops), against per-sample sums written out by hand."""
import bench
from mm_propagation_b200 import workloads as W


def test_merged_terms_join_both_readings_of_a_pair_field():
    prob = W.small_case(M=2)
    prob = prob.replace(coupling=W.nz_array([(0, 0, 0, 1, 1.0), (0, 0, 1, 0, 1.0), (0, 1, 0, 1, 2.0), (1, 0, 1, 0, 0.0),
                                             (1, 1, 1, 1, 3.0)]))
    assert bench.merged_terms(prob) == 3


def test_flops_of_the_forms():
    prob = W.sweep28(seed=0, index=31)
    NT, P, merged = prob.nt, 313, bench.merged_terms(prob)
    assert merged == 1050
    general = bench.stage_flops(prob, P, 2000, 2, True, merged=merged)
    real = bench.stage_flops(prob, P, 2000, 2, True, merged=merged, real=True)
    # a term: x_r = a Re W, x_i = b Im W and four FMAs; real: x = a Re W and two. A pair field: its product (6; 3)
    # and the recurrence (two real inputs of 12 flops; one)
    assert general["contract"] == NT * (10.0 * merged + 6.0 * P + 24.0 * P) and general["pair"] == 24.0 * P * NT
    assert real["contract"] == NT * (5.0 * merged + 3.0 * P + 12.0 * P) and real["pair"] == 12.0 * P * NT


def test_tensor_core_work():
    prob = W.dense15(seed=0, nt=8192)
    # 120 pair fields: 15 chunks of 8; an MMA is 2 x 128 x (16 x 15) x 8 flops a chunk and split term, 64 tiles
    mma = 2.0 * 128 * 240 * 8 * 15 * 3 * 64
    assert bench.tc_mma_flops(prob, 120, real=True) == mma and bench.tc_mma_flops(prob, 120) == 2 * mma
    assert bench.tc_useful_flops(prob, 120, real=True) == (2.0 * 225 * 120 + 4.0 * 225) * 8192
