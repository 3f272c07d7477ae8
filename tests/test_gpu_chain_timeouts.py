"""The cluster chains when the waits for published values run out, made to on
purpose as in test_gpu_timeouts: fronts of 5 blocks (fewer than the cluster has
CTAs), 17 and 18 (past the ring of 16, whose barriers are armed again) and two
fronts side by side.  Every block's result must still reach every CTA of its cluster:
the call reports the timeout, and the solves after it give the same bits as the ones
before.
"""
import numpy as np
import pytest

from tests.helpers import scaled_residual
from tests.test_gpu_front_shapes import blocks_and_separator
from tests.test_gpu_small_solve import star
from tests.test_gpu_timeouts import DEFAULT_LIMIT

SHAPES = [(300, 0, 0), (1080, 0, 0), (1100, 0, 0), (524, 300, 600)]


def matrix(tb, shape):
    s1, s2, m = shape
    return blocks_and_separator(tb, s1, s2, m, seed=sum(shape)) if m else star(tb, 0, 0, s1, seed=s1)


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [1, 8])
@pytest.mark.parametrize("shape", SHAPES, ids=["_".join(map(str, s)) for s in SHAPES])
def test_chains_that_give_up_fp64(tb, shape, nrhs):
    A = matrix(tb, shape)
    B = np.random.default_rng(2).uniform(-1, 1, (A.n, nrhs))
    F = tb.factor_mf(A)
    assert F is not None, tb.last_error()
    for _ in range(3):         # eager, recorded, replayed
        X = F.solve(B)
    assert tb.lib().taucs_b200_debug_waits(2000, 1) == 0
    try:
        with pytest.raises(RuntimeError, match="timed out"):
            F.solve(B)
    finally:
        assert tb.lib().taucs_b200_debug_waits(DEFAULT_LIMIT, 0) == 0
    for _ in range(2):
        assert np.array_equal(F.solve(B), X)
    F.free()


@pytest.mark.gpu
@pytest.mark.parametrize("nrhs", [1, 3, 8])
def test_chains_that_give_up_fp32(tb, nrhs):
    A = matrix(tb, (1100, 0, 0))
    B = np.random.default_rng(2).uniform(-1, 1, (A.n, nrhs))
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    G.set_pcg(0)
    assert G.numeric(A) == 0, tb.last_error()
    X, its, res = G.solve_refine(A, B, tol=1e-12, maxits=10)
    assert 0 <= its <= 4 and res.max() <= 1e-12
    assert tb.lib().taucs_b200_debug_waits(2000, 1) == 0
    try:
        # corrections from values that no tag vouches for (right or wrong): the
        # residual decides, never a wrong answer with success
        Y, its2, res = G.solve_refine(A, B, tol=1e-12, maxits=3)
        assert its2 == -1 or res.max() <= 1e-12
        assert its2 == -1 or max(scaled_residual(A, Y[:, q], B[:, q]) for q in range(nrhs)) <= 1e-12
    finally:
        assert tb.lib().taucs_b200_debug_waits(DEFAULT_LIMIT, 0) == 0
    assert G.numeric(A) == 0, tb.last_error()
    Y, its2, res = G.solve_refine(A, B, tol=1e-12, maxits=10)
    assert its2 == its and res.max() <= 1e-12 and np.array_equal(X, Y)
    G.free()
