"""The one-warp triangular solve of the small fronts (order <= 96) at its
edges: orders around the 32-row slots, panels larger than a warp's slot of
shared memory (taken in pieces), more than 32 children, children in groups,
small fronts above a big one, and every right-hand-side instantiation.  Each
matrix is a dense root of order r with `blocks` dense blocks of order a coupled
to all of it.

* FP64: scaled residual ||A x - b|| / (||A|| ||x|| + ||b||) <= 4 n 2^-53 per
  column (the backward error of a Cholesky solve), also for the
  allocation-free solve.
* FP32 fronts: refinement reaches 1e-12 by FP32 steps alone, at most four of
  them (the matrices are diagonally dominant: a step gains four digits or
  more; a wrong entry of the FP32 solve stalls it).
"""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import scaled_residual

SHAPES = [(0, 0, 1), (0, 0, 31), (0, 0, 32), (0, 0, 33), (0, 0, 65), (0, 0, 96), (40, 3, 50), (5, 20, 33), (2, 48, 48),
          (33, 1, 31), (3, 60, 36), (7, 17, 64), (1, 40, 90), (2, 31, 2)]


def star(tb, blocks, a, r, seed):
    rng = np.random.default_rng(seed)
    n = blocks * a + r
    root = np.arange(blocks * a, n)
    rows, cols = [], []
    for b in range(blocks):
        for j in range(b * a, (b + 1) * a):
            rows.append(np.concatenate([np.arange(j, (b + 1) * a), root]))
            cols.append(np.full(rows[-1].size, j))
    for j in root:
        rows.append(np.arange(j, n))
        cols.append(np.full(rows[-1].size, j))
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    vals = -rng.uniform(0.05, 1.0, rows.size)
    off = rows != cols
    d = np.ones(n)
    np.add.at(d, rows[off], -vals[off])
    np.add.at(d, cols[off], -vals[off])
    vals[~off] = d[rows[~off]]
    cp = np.zeros(n + 1, np.int64)
    np.add.at(cp, cols + 1, 1)
    return tb.Matrix(n, np.cumsum(cp).astype(np.int32), rows.astype(np.int32), vals)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=["_".join(map(str, s)) for s in SHAPES])
def test_small_front_solves(tb, shape):
    import torch
    A = star(tb, *shape, seed=sum(shape))
    B = np.random.default_rng(1).uniform(-1, 1, (A.n, 9))
    bar = 4 * A.n * 2.0 ** -53
    F = tb.factor_mf(A)
    assert F is not None, tb.last_error()
    for nrhs in (1, 2, 3, 4, 5, 8, 9):
        X = F.solve(B[:, :nrhs])
        assert max(scaled_residual(A, X[:, q], B[:, q]) for q in range(nrhs)) <= bar, nrhs
    db = torch.from_numpy(np.ascontiguousarray(B[:, :2].T)).cuda()
    dx = torch.empty_like(db)
    torch.cuda.synchronize()
    assert tb.lib().taucs_b200_solve_device_noalloc(F.h, 2, C.c_void_p(dx.data_ptr()), C.c_void_p(db.data_ptr()),
                                                    A.n) == 0, tb.last_error()
    assert tb.lib().taucs_b200_solve_device_noalloc_status() == 0, tb.last_error()
    X = dx.cpu().numpy()
    assert max(scaled_residual(A, X[q], B[:, q]) for q in range(2)) <= bar
    F.free()
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    assert G.numeric(A) == 0, tb.last_error()
    for nrhs in (1, 3, 8):
        _, its, res = G.solve_refine(A, B[:, :nrhs], tol=1e-12, maxits=10)
        assert 0 <= its <= 4 and res.max() <= 1e-12 and G.refine_report()[0] == 0, (nrhs, its, res)
    G.free()
