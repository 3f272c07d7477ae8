"""The FP64 products' tile shapes on fronts either side of the line between
32x32 and 64x64 tiles (four waves of 64x64 tiles, 1776) and with the 128x128 variant:
two update matrices of 16, 17, 2560 (1640 tiles) and 2688 (1806) rows from panels of 130 columns (a panel
product and remainders of every tile), against NumPy's Cholesky of the same
dense matrix, within 100 n 2^-53 (relative Frobenius; c n u |L| with c < 100 for
these diagonally dominant matrices).
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import blocks_and_separator
from tests.test_gpu_panel import dense_l, dominant, full


@pytest.mark.gpu
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("m", [16, 17, 2560, 2688])
def test_gemm_tiles(tb, m, variant):
    A = blocks_and_separator(tb, 130, 100, m, seed=m)
    n, cp, ri, _ = A.arrays()
    A = tb.Matrix(n, cp, ri, dominant(A))
    F = tb.factor_symbolic(A)
    F.set_gemm_choices(0, [variant] * (2 * F.info().n_levels))
    assert F.numeric(A) == 0, tb.last_error()
    ref = np.linalg.cholesky(full(A))
    assert np.linalg.norm(dense_l(tb, F, n) - ref) <= 100 * n * 2.0 ** -53 * np.linalg.norm(ref)
    F.free()
