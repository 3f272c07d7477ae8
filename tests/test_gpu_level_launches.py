"""Panel steps and products over a level of many fronts of different sizes (each
launch's CTAs are counted front by front): 33, 40 and 70 dense blocks of 97 to
300 columns, coupled to one dense root block of 40 rows, so that the number of
fronts falls from step to step and is on both sides of one search round (32);
30 blocks with a root block of 577 and 640 rows, for which FP32 steps take row
CTAs of 256 rows (two waves of 64 rows, one of 256), the last one not full.
FP64 against NumPy's Cholesky, FP32 fronts against FP64's factor of the scaled
matrix; bars as in test_gpu_panel (100 n 2^-53 and 100 n 2^-24, relative
Frobenius, diagonally dominant matrices).
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import _scaled
from tests.test_gpu_panel import dense_l, full


def blocks(tb, count, r, seed):
    rng = np.random.default_rng(seed)
    sizes = rng.integers(97, 141, count)
    sizes[:3] = 300, 257, 128
    rng.shuffle(sizes)
    n = int(sizes.sum()) + r
    root = np.arange(n - r, n)
    rows, lo = [], 0
    for a in sizes:
        rows += [np.concatenate([np.arange(j, lo + a), root]) for j in range(lo, lo + a)]
        lo += a
    rows += [np.arange(j, n) for j in root]
    cols = np.concatenate([np.full(x.size, j) for j, x in enumerate(rows)])
    rows = np.concatenate(rows)
    vals = -rng.uniform(0.05, 1.0, rows.size)
    off = rows != cols
    d = np.ones(n)
    np.add.at(d, rows[off], -vals[off])
    np.add.at(d, cols[off], -vals[off])
    vals[~off] = 2.0 * d[rows[~off]]
    cp = np.zeros(n + 1, np.int64)
    np.add.at(cp, cols + 1, 1)
    return tb.Matrix(n, np.cumsum(cp).astype(np.int32), rows.astype(np.int32), vals)


@pytest.mark.gpu
@pytest.mark.parametrize("count, root", [(33, 40), (40, 40), (70, 40), (30, 577), (30, 640)])
def test_levels_of_many_fronts(tb, count, root):
    A = blocks(tb, count, root, seed=count)
    n, cp, ri, _ = A.arrays()
    F = tb.factor_symbolic(A)
    assert F.numeric(A) == 0, tb.last_error()
    ref = np.linalg.cholesky(full(A))
    assert np.linalg.norm(dense_l(tb, F, n) - ref) <= 100 * n * 2.0 ** -53 * np.linalg.norm(ref)
    F.free_numeric()
    assert F.numeric(tb.Matrix(n, cp, ri, _scaled(A))) == 0, tb.last_error()
    _, ref = F.export_values()
    F.free()
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    assert G.numeric(A) == 0, tb.last_error()
    _, got = G.export_values()
    assert np.linalg.norm(got - ref) <= 100 * n * 2.0 ** -24 * np.linalg.norm(ref)
    G.free()
