"""The triangular solves of big fronts at the edges of the cluster chains and
of the block kernels: chains of 4 blocks (the shortest), of fewer blocks than
the cluster has CTAs, one more, more than two turns; last blocks of 1, 12 and
63 columns with update rows in them; none, one and two chunks of 512 update
rows; two fronts of different length side by side; and chains just below the
limit, which the block kernels take.

Matrices as in test_gpu_front_shapes (two dense blocks, a dense separator, a
dense top block), or one dense front.  FP64: scaled residual <= 4 n 2^-53 per
column (the backward error of a Cholesky solve).  FP32 fronts: refinement
reaches 1e-12 by at most four FP32 steps (diagonally dominant matrices: four
digits a step or more; a wrong entry of the FP32 solve stalls it).
"""
import numpy as np
import pytest

from tests.helpers import scaled_residual
from tests.test_gpu_front_shapes import blocks_and_separator
from tests.test_gpu_small_solve import star

SHAPES = [(256, 0, 0), (255, 0, 0), (300, 0, 0), (513, 0, 0), (577, 0, 0), (1100, 0, 0), (257, 300, 130),
          (524, 140, 600), (319, 128, 513), (200, 250, 90)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=["_".join(map(str, s)) for s in SHAPES])
def test_big_front_solves(tb, shape):
    s1, s2, m = shape
    A = blocks_and_separator(tb, s1, s2, m, seed=sum(shape)) if m else star(tb, 0, 0, s1, seed=s1)
    B = np.random.default_rng(1).uniform(-1, 1, (A.n, 9))
    bar = 4 * A.n * 2.0 ** -53
    F = tb.factor_mf(A)
    assert F is not None, tb.last_error()
    for nrhs in (1, 2, 3, 4, 8, 9):
        for _ in range(3):     # eager, recorded, replayed
            X = F.solve(B[:, :nrhs])
        assert max(scaled_residual(A, X[:, q], B[:, q]) for q in range(nrhs)) <= bar, nrhs
    F.free()
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    assert G.numeric(A) == 0, tb.last_error()
    for nrhs in (1, 3, 8):
        _, its, res = G.solve_refine(A, B[:, :nrhs], tol=1e-12, maxits=10)
        assert 0 <= its <= 4 and res.max() <= 1e-12 and G.refine_report()[0] == 0, (nrhs, its, res)
    G.free()
