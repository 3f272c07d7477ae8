"""Every entry of FP32 factors, in both split formats of the tensor-core products: the
row CTAs of 64, 128 and 256 rows, levels of many fronts, and single dense fronts.  A
norm over a whole factor cannot see a CTA that was left out (its share of a large
factor's norm is under any bar of n 2^-24), so each entry of L L^T - A is held against
its own bound, g (|L| |L|^T), A the scaled matrix that FP32 fronts factor.

g = (4 k + 64) 2^-24 for an entry that sums k products (Higham, Accuracy and Stability of
Numerical Algorithms, theorem 10.3, has (k + 1) u): the accumulators of the tensor cores
truncate (2 u a sum); a split product is off by 3 x 2^-22 = 12 u (two parts of 11 bits
each: what the lower part rounds off each operand, and lo lo left out), and with FP16
parts by another 2^-36 absolute for entries below 2^-14 (42 u at the smallest here,
2^-16.4); the pivots' reciprocal square roots by a few u, the scaled matrix by u.
Together 2 k + 64 and some, with k >= 97: half of g.  An entry that was left out is off
by its own size, 10^3 to 10^4 times its bound.
"""
import numpy as np
import pytest

from tests.test_gpu_front_shapes import _scaled, blocks_and_separator
from tests.test_gpu_level_launches import blocks
from tests.test_gpu_panel import BELOW, dominant
from tests.test_gpu_small_solve import star

SHAPES = ([("blocks", c, r) for c, r in [(33, 40), (70, 40), (30, 577), (30, 640)]] + [("below", *s) for s in BELOW]
          + [("dense", s) for s in (97, 129, 145, 257, 385)])


def matrix(tb, shape):
    kind, *s = shape
    if kind == "blocks":
        return blocks(tb, *s, seed=s[0])
    A = blocks_and_separator(tb, *s, seed=sum(s)) if kind == "below" else star(tb, 0, 0, s[0], seed=s[0])
    n, cp, ri, _ = A.arrays()
    return tb.Matrix(n, cp, ri, dominant(A))


def worst(G, A):
    """Largest |L L^T - A| / (g |L| |L|^T) over the entries of L's pattern: fronts whose
    update rows all belong to one root."""
    n, cp, ri, _ = A.arrays()
    va = _scaled(A)
    sym = G.export_symbolic()
    vp, v = G.export_values()
    fronts = []
    for i in range(sym["n_sn"]):
        s, f = int(sym["sn_size"][i]), int(sym["sn_up_size"][i])
        if vp[i + 1] > vp[i]:
            rows = sym["struct_idx"][sym["struct_ptr"][i]:sym["struct_ptr"][i] + f]
            P = v[vp[i]:vp[i + 1]].reshape(s, f).T.copy()
            P[:s] = np.tril(P[:s])
            fronts.append((rows, s, P))
    roots = [F for F in fronts if F[0].size == F[1]]
    rrows, rs, _ = roots[-1]
    at = np.full(n, -1)
    at[rrows] = np.arange(rs)
    S, M = np.zeros((rs, rs)), np.zeros((rs, rs))
    bad = 0.0
    for rows, s, P in sorted(fronts, key=lambda F: F[0] is rrows):
        lp, mp, k = P @ P[:s].T, np.abs(P) @ np.abs(P[:s]).T, s
        if rows is rrows:
            lp, mp, k = lp + S, mp + M, n
        elif rows.size > s:
            u = at[rows[s:]]
            assert (u >= 0).all()
            S[np.ix_(u, u)] += P[s:] @ P[s:].T
            M[np.ix_(u, u)] += np.abs(P[s:]) @ np.abs(P[s:]).T
        order = np.argsort(rows)
        for j in range(s):
            c = rows[j]
            e = np.arange(cp[c], cp[c + 1])
            lp[order[np.searchsorted(rows, ri[e], sorter=order)], j] -= va[e]
        low = rows[:, None] >= rows[None, :s]
        g = (4 * k + 64) * 2.0 ** -24
        bad = max(bad, float((np.abs(lp) / np.where(mp > 0, g * mp, 1.0))[low].max()))
    return bad


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", [0, 1], ids=["tf32", "fp16"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "_".join(map(str, s)))
def test_every_entry_of_fp32_factors(tb, shape, fmt):
    A = matrix(tb, shape)
    G = tb.factor_symbolic(A)
    G.set_precision(1)
    tb.lib().taucs_b200_set_split_format(G.h, fmt)
    for _ in range(3):         # eager, recorded, replayed
        assert G.numeric(A) == 0, tb.last_error()
    assert worst(G, A) <= 1.0
    G.free()


@pytest.mark.parametrize("shape", [("blocks", 30, 577), ("below", 300, 200, 129), ("dense", 385)],
                         ids=lambda s: "_".join(map(str, s)))
def test_the_bound_sees_what_it_should(tb, shape):
    """Host: the exact factor rounded to FP32 passes; with a 16 x 16 tile of it, or one
    entry, off by a hundredth it does not."""
    A = matrix(tb, shape)
    G = tb.factor_symbolic(A)
    n, cp, ri, _ = A.arrays()
    sym = G.export_symbolic()
    D = np.zeros((n, n))
    D[ri, np.repeat(np.arange(n), np.diff(cp))] = _scaled(A)
    L = np.linalg.cholesky(D + np.tril(D, -1).T)
    vp, parts = [0], []
    for i in range(sym["n_sn"]):
        s, f = int(sym["sn_size"][i]), int(sym["sn_up_size"][i])
        rows = sym["struct_idx"][sym["struct_ptr"][i]:sym["struct_ptr"][i] + f]
        parts.append(L[np.ix_(rows, rows[:s])].T.ravel())
        vp.append(vp[-1] + s * f)

    class Export:
        def export_symbolic(self):
            return sym

        def export_values(self):
            return np.array(vp), self.v

    E = Export()
    E.v = np.concatenate(parts).astype(np.float32).astype(np.float64)
    assert worst(E, A) <= 1.0
    i = int(np.argmax(np.diff(vp)))
    s, f = int(sym["sn_size"][i]), int(sym["sn_up_size"][i])
    good = E.v[vp[i]:vp[i + 1]].reshape(s, f).copy()
    for r0, r1, c0, c1 in [(f - 16, f, 64, 80), (f - 16, f, s - 16, s), (f - 1, f, 0, 1)]:
        P = good.copy()
        P[c0:c1, r0:r1] *= 0.99
        E.v[vp[i]:vp[i + 1]] = np.where(np.arange(f)[None, :] >= np.arange(s)[:, None], P, 0.0).ravel()
        assert worst(E, A) > 1.0, (r0, c0)
    G.free()
