"""The flop model of a solve's level-0 kernels against operation counts of the
loops written out for the smallest shape, D = 2, d = 1 (a multiply-add is 2)."""

from pof import _flops


def test_solve_level0_counts_what_a_solve_runs():
    # no filter objective in a solve, structured at every D
    for D, d in ((2, 1), (3, 1), (4, 1), (4, 2), (5, 1), (6, 2), (8, 2), (12, 3)):
        C0, cnt = _flops.plan_levels(1000, D)
        assert _flops.kernel_flops("filt_l0_down", 1000, D, d, C0, cnt) == 1000 * _flops.kf_step(D, d, True, True)
        assert _flops.kf_step(D, d, True, True) < _flops.kf_step(D, d, True, False)
        assert _flops.cond_fold_step(D, d, True) < _flops.cond_fold_step(D, d, False)


def test_counts_at_the_smallest_shape():
    # lq of [QL | F L], one nonzero column: per reflector 2 |x|^2, 8 scalars, 7 per row below
    assert _flops.lq(2, lambda j: 1) == (2 + 8 + 7) + (2 + 8)
    # E g1 (8) + g2 (2), E2 D1 (one column: 4 multiply-adds = 8), [D2 | .] (27), E2 E1 (16)
    assert _flops.l0_smooth_combine(2, 1) == 8 + 2 + 8 + 27 + 16
    # E m (8) + g (2), E L (6 multiply-adds = 12), tails of 2 and 1: (4 + 8 + 11) + (2 + 8)
    assert _flops.l0_smooth_apply(2, 1) == 8 + 2 + _flops.mm_lowerB(2, 2) + 23 + 10
