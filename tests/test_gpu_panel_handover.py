"""The hand-over inside a panel step, from the CTA that factors a front's diagonal
block to the CTAs that hold the rows below it: those rows follow a counter piece by
piece, some pieces fetched ahead and some waited for, which changes from run to run
and must not show in the result.  A front of 300 columns (three steps, the last of 44)
over 1500 rows, in 12 (128 rows) to 24 (64) row CTAs, factored again and again:
the same bits each time, and each column block's residual within the
componentwise bound of a Cholesky factor, |L L^T - A| <= g |L| |L|^T with g = 2 (k + 8)
2^-53, k the number of products that an entry sums (Higham, Accuracy and Stability of
Numerical Algorithms, theorem 10.3: (k + 1) u; 8 for the reciprocal pivots; twice, since
the check's own product rounds as much).
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import blocks_and_separator
from tests.test_gpu_panel import dense_l, full


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_rows_follow_the_diagonal_block(tb, prec):
    A = blocks_and_separator(tb, 300, 100, 1500, seed=5)
    F = tb.factor_symbolic(A)
    F.set_precision(prec)
    assert F.numeric(A) == 0, tb.last_error()
    vp, first = F.export_values()
    for _ in range(20):
        assert F.numeric(A) == 0, tb.last_error()
        assert np.array_equal(F.export_values()[1], first)
    if prec == 0:
        # the first block's columns: only their own products, rows of the block and the separator
        a = full(A)
        l = dense_l(tb, F, A.n)[:, :300]
        rows = np.r_[0:300, 400:1900]
        r = np.abs(l[rows] @ l[:300].T - a[rows, :300])
        assert (r <= 2 * (300 + 8) * 2.0 ** -53 * (np.abs(l[rows]) @ np.abs(l[:300]).T)).all()
    F.free()
