"""The hand-over inside a panel step, from the CTA that factors a front's diagonal
block to the CTAs that hold the rows below it: those rows follow a counter piece by
piece, some pieces fetched ahead and some waited for, which changes from run to run
and must not show in the result.  Two fronts of 300 columns (three steps, the last of
44) over 1300 rows, in 11 row CTAs of 128 rows each, factored again and again: the same
bits each time, and the first block's residual within the componentwise bound of a
Cholesky factor, |L L^T - A| <= g |L| |L|^T with g = 2 (k + 8) 2^-53, k the number of
products that an entry sums (Higham, Accuracy and Stability of Numerical Algorithms,
theorem 10.3: (k + 1) u; 8 for the reciprocal pivots; twice, since the check's own
product rounds as much).
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import blocks_and_separator
from tests.test_gpu_level_launches import blocks
from tests.test_gpu_panel import dense_l, full


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
def test_rows_follow_the_diagonal_block(tb, prec):
    A = blocks_and_separator(tb, 300, 300, 1300, seed=5)
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
        rows = np.r_[0:300, 600:1900]
        r = np.abs(l[rows] @ l[:300].T - a[rows, :300])
        assert (r <= 2 * (300 + 8) * 2.0 ** -53 * (np.abs(l[rows]) @ np.abs(l[:300]).T)).all()
    F.free()


def indefinite(A, col):
    """A with a diagonal entry (of a column coupled to earlier ones) so small, but
    positive, that its pivot is the first nonpositive one (the leading minors
    before it are A's): FP32 fronts pass the scaling and fail in the panel."""
    n, cp, ri, va = A.arrays()
    v = va.copy()
    assert ri[cp[col]] == col
    v[cp[col]] = 1e-6
    return type(A)(n, cp, ri, v)


def fails_at(tb, F, A, col):
    """The factorization fails and names the column: a wait that ran out would
    have replaced it (and kept FP32 fronts from falling back to FP64)."""
    bad = indefinite(A, col)
    for _ in range(3):         # eager, recorded, replayed
        assert F.numeric(bad) != 0
        assert "LL^T Factorization" in tb.last_error()
        assert f"(nonpositive pivot in column {col})" in tb.last_error(), tb.last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("col", [1, 16, 127, 128, 250, 299, 1300])
def test_failing_front_releases_the_rows_below(tb, col, prec):
    """The first and last pieces of each step, in one of two fronts of 300
    columns over 1300 rows and (column 1300) in the root above them."""
    A = blocks_and_separator(tb, 300, 300, 1300, seed=5)
    F = tb.factor_symbolic(A)
    F.set_precision(prec)
    fails_at(tb, F, A, col)
    assert F.numeric(A) == 0, tb.last_error()
    F.free()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("count, root", [(70, 40), (30, 640)])
def test_one_failing_front_among_many(tb, count, root, prec):
    """A level of many fronts of which one fails, early or late in the launch's
    list (sorted by columns) and in the first or second step; the others' rows
    follow their own diagonal blocks meanwhile."""
    A = blocks(tb, count, root, seed=count)
    n, cp, ri, _ = A.arrays()
    # each leaf block's first column: its rows run to the block's end, then the root
    first, j = [], 0
    while j < n - root:
        first.append(j)
        j += int((ri[cp[j]:cp[j + 1]] < n - root).sum())
    size = np.diff(np.r_[first, n - root])
    F = tb.factor_symbolic(A)
    F.set_precision(prec)
    assert F.numeric(A) == 0, tb.last_error()
    good = F.export_values()[1]
    widest = int(np.argmax(size))
    for blk, off in [(0, 5), (count // 2, 60), (count - 1, 96), (widest, 20), (widest, 200)]:
        fails_at(tb, F, A, first[blk] + off)
        assert F.numeric(A) == 0, tb.last_error()
        assert np.array_equal(F.export_values()[1], good)
    F.free()
