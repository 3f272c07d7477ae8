"""The 128-column panel steps at their edges: one front of s columns (pieces of
16: s on, below and above a multiple of 16; one step, one column more, two steps,
two and one column) and fronts with 1, 63..65 and 127..129 rows below the last
step (the row CTAs hold 64 or 128), against NumPy's Cholesky of the same dense
matrix.

Matrices: strictly diagonally dominant by a factor (condition number < 100), so
each Cholesky is within c n u |L| of the exact one with c < 100 (normwise); the
bars are 100 n 2^-53 in FP64 and, for the scaled matrix that FP32 fronts hold, 100
n 2^-24 on L (relative Frobenius).  A pivot that is not positive, in the first
or a later piece or step, fails the factorization, and the next one on the same
factor object works.
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import _scaled, blocks_and_separator
from tests.test_gpu_small_solve import star

DENSE = [97, 111, 112, 113, 127, 128, 129, 144, 145, 255, 256, 257, 385]
BELOW = [(97, 100, 1), (128, 130, 63), (113, 128, 64), (257, 127, 65), (129, 145, 127), (100, 98, 128), (300, 200, 129)]


def full(A):
    n, cp, ri, va = A.arrays()
    D = np.zeros((n, n))
    D[ri, np.repeat(np.arange(n), np.diff(cp))] = va
    return D + np.tril(D, -1).T


def dominant(A):
    """Twice the diagonal: every eigenvalue within a factor of three of it."""
    n, cp, ri, va = A.arrays()
    v = va.copy()
    v[ri == np.repeat(np.arange(n), np.diff(cp))] *= 2.0
    return v


def dense_l(tb, F, n):
    L = F.to_ccs()
    _, cp, ri, va = L.arrays()
    D = np.zeros((n, n))
    D[ri, np.repeat(np.arange(n), np.diff(cp))] = va
    return D


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(s, 0, 0) for s in DENSE] + BELOW, ids=lambda s: "_".join(map(str, s)))
def test_panel_shapes(tb, shape):
    s1, s2, m = shape
    A = blocks_and_separator(tb, s1, s2, m, seed=sum(shape)) if m else star(tb, 0, 0, s1, seed=s1)
    n, cp, ri, _ = A.arrays()
    A = tb.Matrix(n, cp, ri, dominant(A))
    F = tb.factor_symbolic(A)
    for _ in range(3):         # eager, recorded, replayed
        assert F.numeric(A) == 0, tb.last_error()
    got, ref = dense_l(tb, F, n), np.linalg.cholesky(full(A))
    assert np.linalg.norm(got - ref) <= 100 * n * 2.0 ** -53 * np.linalg.norm(ref)
    # FP32 fronts hold the factor of D A D, D = diag(A)^-1/2: against FP64's of it
    F.free_numeric()
    assert F.numeric(tb.Matrix(n, cp, ri, _scaled(A))) == 0, tb.last_error()
    _, ref = F.export_values()
    F.free()
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    for _ in range(3):
        assert G.numeric(A) == 0, tb.last_error()
    _, got = G.export_values()
    assert np.linalg.norm(got - ref) <= 100 * n * 2.0 ** -24 * np.linalg.norm(ref)
    G.free()


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("col", [0, 15, 16, 100, 127, 128, 150, 255])
def test_panel_nonpositive_pivot(tb, col, prec):
    A = star(tb, 0, 0, 256, seed=3)
    n, cp, ri, va = A.arrays()
    bad = va.copy()
    bad[cp[col]] = -1.0
    F = tb.factor_symbolic(A)
    F.set_precision(prec)
    for _ in range(2):
        assert F.numeric(tb.Matrix(n, cp, ri, bad)) != 0
        assert F.numeric(A) == 0, tb.last_error()
    b = np.ones(n)
    x = F.solve(b)
    bar = 4 * n * (2.0 ** -20 if prec else 2.0 ** -53)
    assert np.abs(A.matvec(x) - b).max() <= bar * (A.inf_norm() * np.abs(x).max() + 1)
    F.free()
