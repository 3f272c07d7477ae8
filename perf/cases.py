"""The work that programs have this library do, as timed cases.

A case is one call sequence of a user's program through the Python mirror of
the C interface, on a finite-difference operator with lognormal edge
conductances (the matrices of the benchmark, the request stream and the
batches: 5-point grids in 2D, 7-point grids in 3D, Dirichlet boundary):

  step      new values on an analysed pattern: numeric factorization, then the
            solution (FP64: triangular solves; mixed: FP32 fronts and FP64
            refinement to a scaled residual of `tol`)
  solve     triangular solves with a factor that is already there (FP64)
  refine    refined solutions with an FP32 factor that is already there
  batch     new values for many small systems analysed as one: factorization
            and refinement of all of them, one right-hand side each
  linsolve  one call of taucs_linsolve on host arrays: ordering, symbolic
            analysis, factorization and solution

`data` says where the program holds values and vectors: in device memory, or
in host arrays handed to the C interface as they are.  Right-hand sides and
solutions are in the grid's own order, as a program holds them; the fill-
reducing permutation is applied around the call.

The request server is not timed on its own: its requests are the mixed steps
and refinements below, in an order among its workers that differs from run to
run.
"""
import numpy as np
import torch

import taucs_b200 as tb

LLT_OPTIONS = ["taucs.factor.LLT=true", "taucs.factor.mf=true", "taucs.factor.ordering=amd"]
LLT_MIXED = LLT_OPTIONS + ["taucs.gpu.precision=mixed", "taucs.gpu.refine.tol=1e-13"]
MAXITS = 10


def _case(name, kind, x, y, z, precision, nrhs, data, sigma=1.0, aniso=1.0, tol=1e-13):
    c = dict(kind=kind, x=x, y=y, z=z, precision=precision, nrhs=nrhs, data=data, sigma=sigma, aniso=aniso, tol=tol)
    return dict(c, name=name) if name else c


def _batch(name, count, precision, tol=1e-13):
    c = dict(kind="batch", count=count, precision=precision, sigma=1.0, tol=tol)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one right-hand side on a resident 2D factor, from and to host arrays
        _case("solve_2d_33_host", "solve", 33, 33, 0, "fp64", 1, "host"),
        # the reference's own acceptance size (2D, 100 a side): refactor and solve from host arrays
        _case("step_2d_100_fp64_host", "step", 100, 100, 0, "fp64", 1, "host"),
        # a 2D request of the served mix (1k to 20k unknowns), ragged sides
        _case("step_2d_139x142_mixed", "step", 139, 142, 0, "mixed", 1, "device"),
        # a small 3D request of the served mix (16 to 40 a side), ragged, an odd number of right-hand sides
        _case("step_3d_29x24x26_mixed", "step", 29, 24, 26, "mixed", 3, "device"),
        # an ordinary 3D system in full precision: a nonlinear or time-stepping program's refactor and solve
        _case("step_3d_40x41x39_fp64", "step", 40, 41, 39, "fp64", 1, "device"),
        # the FP64 benchmark size
        _case("step_3d_64_fp64", "step", 64, 64, 64, "fp64", 1, "device"),
        # the precision benchmark: 80 a side, strongly varying and anisotropic, 8 right-hand sides
        _case("step_3d_80_mixed", "step", 80, 80, 80, "mixed", 8, "device", sigma=2.0, aniso=100.0),
        # time stepping with a constant matrix: one right-hand side after another on a resident factor
        _case("solve_3d_64_fp64", "solve", 64, 64, 64, "fp64", 1, "device"),
        # many right-hand sides at once (up to 32 a request), ragged sides
        _case("solve_3d_45x47x44_fp64_r32", "solve", 45, 47, 44, "fp64", 32, "device"),
        # a request for a matrix that is factored already: refinement only
        _case("refine_3d_56_mixed_r8", "refine", 56, 56, 56, "mixed", 8, "device"),
        # many small independent systems, 2D of 8 to 96 and 3D of 4 to 24 a side
        _batch("batch_512_mixed", 512, "mixed"),
        # a one-shot program: everything from the unordered host matrix on
        _case("linsolve_3d_20", "linsolve", 20, 20, 20, "fp64", 1, "host"),
    ]


def _log_uniform(rng, lo, hi):
    return float(lo) * (float(hi) / float(lo)) ** rng.random()


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "solve", "refine", "batch", "linsolve"])
    if kind == "batch":
        return _batch(None, int(_log_uniform(rng, 24, 768)), rng.choice(["mixed", "fp64"]))
    precision = {"solve": "fp64", "refine": "mixed"}.get(kind) or rng.choice(["fp64", "mixed"])
    flat = rng.random() < 0.35
    data = rng.choice(["device", "device", "host"])
    nrhs = rng.choice([1, 1, 1, 2, 3, 5, 8])
    if kind == "linsolve":
        n, data, nrhs = _log_uniform(rng, 500, 12000), "host", rng.choice([1, 1, 4])
    elif flat:
        n = _log_uniform(rng, 1000, 120000)
    else:
        n = _log_uniform(rng, 1000, 400000 if precision == "mixed" else 230000)
        if kind == "solve" and n < 120000:
            nrhs = rng.choice([1, 1, 4, 8, 19, 32])
    stretch = [rng.uniform(0.75, 1.3) for _ in range(2 if flat else 3)]
    side = (n / float(np.prod(stretch))) ** (1.0 / len(stretch))
    dims = [max(3, int(round(side * s))) for s in stretch]
    x, y, z = dims + [0] if flat else dims
    sigma, aniso = rng.choice([(1.0, 1.0), (1.0, 1.0), (0.5, 10.0), (2.0, 100.0)])
    return _case(None, kind, x, y, z, precision, nrhs, data, sigma=sigma, aniso=aniso)


# ------------------------------------------------------------------ inputs


class Grid:
    """Conductances of an X x Y x Z grid (Z = 0: X x Y): exp(sigma N(0,1)), the last axis times `aniso`, boundary
    faces included and added to the diagonal."""

    def __init__(self, x, y, z, sigma, aniso, rng):
        self.dims = (x, y, z) if z > 0 else (x, y)
        self.n = int(np.prod(self.dims))
        self.edges = []
        self.diag = np.zeros(self.dims)
        for ax in range(len(self.dims)):
            shape = list(self.dims)
            shape[ax] += 1
            c = np.exp(sigma * rng.standard_normal(shape)) * (aniso if ax == len(self.dims) - 1 else 1.0)
            lo = [slice(None)] * len(shape)
            hi = [slice(None)] * len(shape)
            lo[ax], hi[ax] = slice(0, -1), slice(1, None)
            self.diag += c[tuple(lo)] + c[tuple(hi)]
            inner = [slice(None)] * len(shape)
            inner[ax] = slice(1, -1)
            self.edges.append(np.ascontiguousarray(c[tuple(inner)]))

    def lower(self):
        """The lower triangle by columns (rows ascending), as the library takes it."""
        nd = len(self.dims)
        strides = [int(np.prod(self.dims[ax + 1:])) for ax in range(nd)]
        cols = np.arange(self.n, dtype=np.int64).reshape(self.dims)
        vals, rows, keep = [self.diag.reshape(-1)], [cols.reshape(-1)], [np.ones(self.n, bool)]
        for ax in reversed(range(nd)):
            v, k = np.zeros(self.dims), np.zeros(self.dims, bool)
            at = [slice(None)] * nd
            at[ax] = slice(0, -1)
            v[tuple(at)] = -self.edges[ax]
            k[tuple(at)] = True
            vals.append(v.reshape(-1))
            rows.append((cols + strides[ax]).reshape(-1))
            keep.append(k.reshape(-1))
        keep = np.stack(keep, 1)
        colptr = np.zeros(self.n + 1, np.int32)
        np.cumsum(keep.sum(1), out=colptr[1:])
        return tb.Matrix(self.n, colptr, np.stack(rows, 1)[keep].astype(np.int32), np.stack(vals, 1)[keep])


def _inputs(case, seed):
    rng = np.random.default_rng([seed, case["x"], case["y"], case["z"]])
    g = Grid(case["x"], case["y"], case["z"], case["sigma"], case["aniso"], rng)
    return g, rng.uniform(-1.0, 1.0, (case["nrhs"], g.n))      # one row a right-hand side: column-major n x nrhs


def _batch_inputs(case, seed):
    """Half 2D, half 3D grids; the sizes depend on the count alone, values and right-hand sides on the seed."""
    sizes = np.random.default_rng([11, case["count"]])
    grids, bs = [], []
    for i in range(case["count"]):
        two = i < case["count"] // 2
        k = int(sizes.integers(8, 97)) if two else int(sizes.integers(4, 25))
        rng = np.random.default_rng([seed, i])
        grids.append(Grid(k, k, 0 if two else k, case["sigma"], 1.0, rng))
        bs.append(rng.uniform(-1.0, 1.0, grids[-1].n))
    return grids, bs


# ------------------------------------------------------------------ the calls


def _ok(good):
    if not good:
        raise RuntimeError("taucs_b200: " + tb.last_error())


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.kind, s.mixed = case, case["kind"], case["precision"] == "mixed"
    if s.kind == "batch":
        grids, bs = _batch_inputs(case, seed)
        s.F = tb.Batch([g.lower() for g in grids])
        offs = np.concatenate([[0], np.cumsum([g.n for g in grids])])
        perm = s.F.combined_rhs([np.arange(offs[i], offs[i + 1], dtype=np.float64) for i in range(len(grids))])
        s.n, s.nrhs, s.data = s.F.n, 1, "device"
        s.perm = torch.from_numpy(perm.astype(np.int64)).cuda()
        s.values = torch.from_numpy(s.F.combined_values()).cuda()
        s.b = torch.from_numpy(np.concatenate(bs)[None]).cuda()
    else:
        g, b = _inputs(case, seed)
        s.n, s.nrhs, s.data = g.n, case["nrhs"], case["data"]
        A = g.lower()
        if s.kind == "linsolve":
            s.A = A
            s.B = np.asfortranarray(b.T)
            s.X = np.zeros_like(s.B, order="F")
            return s
        perm, iperm = tb.order(A, "amd")
        s.P = A.permute(perm, iperm)
        s.F = tb.factor_symbolic(s.P)
        if s.data == "host":
            s.perm, s.b = perm, b
        else:
            s.perm = torch.from_numpy(perm.astype(np.int64)).cuda()
            s.values = torch.from_numpy(s.P.values).cuda()
            s.b = torch.from_numpy(b).cuda()
    if s.mixed:
        s.F.set_precision(1)
    if s.data == "device":
        s.iperm = torch.empty_like(s.perm)
        s.iperm[s.perm] = torch.arange(s.n, device="cuda")
        s.bp, s.xp, s.x = torch.empty_like(s.b), torch.empty_like(s.b), torch.empty_like(s.b)
    if s.kind in ("solve", "refine"):
        _factor(s)
    return s


def _factor(s):
    if s.data == "host":
        _ok(s.F.numeric(s.P) == 0)
    else:
        _ok(s.F.numeric_device(s.values.data_ptr()) == 0)


def _solve_host(s):
    bp = s.b[:, s.perm]
    x = np.empty_like(bp)
    if s.mixed:
        xp, its, _ = s.F.solve_refine(s.P, bp[0] if s.nrhs == 1 else bp.T, s.case["tol"], MAXITS)
        _ok(its >= 0)
    else:
        xp = s.F.solve(bp[0] if s.nrhs == 1 else bp.T)
    x[:, s.perm] = xp.T
    return x


def _solve_device(s):
    torch.index_select(s.b, 1, s.perm, out=s.bp)
    if s.mixed:
        its, _ = s.F.solve_refine_device(s.nrhs, s.xp.data_ptr(), s.bp.data_ptr(), s.n, s.case["tol"], MAXITS)
        _ok(its >= 0)
    else:
        _ok(s.F.solve_device(s.nrhs, s.xp.data_ptr(), s.bp.data_ptr(), s.n) == 0)
    torch.index_select(s.xp, 1, s.iperm, out=s.x)
    return s.x


def run(s):
    if s.kind == "linsolve":
        F = [None]
        _ok(tb.linsolve(s.A, F, s.nrhs, s.X, s.B, LLT_MIXED if s.mixed else LLT_OPTIONS) == 0)
        tb.linsolve(None, F, 0, None, None, [])      # frees the factor
        return s.X
    if s.kind in ("step", "batch"):
        _factor(s)
    return _solve_host(s) if s.data == "host" else _solve_device(s)


# ------------------------------------------------------------------ what a pass cannot do without


def work(case):
    if case["kind"] == "batch":
        F = tb.Batch([g.lower() for g in _batch_inputs(case, 0)[0]])
        n, nnz, nrhs = F.n, F.nnz, 1
    else:
        A = _inputs(dict(case, nrhs=1), 0)[0].lower()
        n, nnz, nrhs = A.n, A.nnz, case["nrhs"]
        F = tb.factor_symbolic(A.permute(*tb.order(A, "amd")))
    fr, _ = F.layout()
    sz, order = fr[:, 2].astype(np.float64), fr[:, 3].astype(np.float64)
    nnz_l = float(np.sum(sz * order - sz * (sz - 1) / 2))
    esz = 4.0 if case["precision"] == "mixed" else 8.0
    # the factor written (or read) once, the vectors read and written once, the values read once
    nbytes = esz * nnz_l + 16.0 * n * nrhs
    flops = 4.0 * nnz_l * nrhs
    if case["kind"] in ("step", "batch", "linsolve"):
        nbytes += 8.0 * nnz
        flops += float(F.info().flops)
    elif case["kind"] == "refine":
        nbytes += 8.0 * nnz
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ the same results in 64 bits, by other means


def _exact_dense(g, b):
    n = g.n
    cols = np.arange(n).reshape(g.dims)
    A = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    A.diagonal().copy_(torch.from_numpy(g.diag.reshape(-1)))
    for ax, e in enumerate(g.edges):
        i = torch.from_numpy(np.take(cols, range(g.dims[ax] - 1), ax).reshape(-1)).cuda()
        j = torch.from_numpy(np.take(cols, range(1, g.dims[ax]), ax).reshape(-1)).cuda()
        v = -torch.from_numpy(e.reshape(-1)).cuda()
        A[i, j] = v
        A[j, i] = v
    C = torch.linalg.cholesky(A)
    B = torch.from_numpy(b.T.copy()).cuda()
    X = torch.cholesky_solve(B, C)
    X += torch.cholesky_solve(B - A @ X, C)
    return X.T.contiguous()


def _exact_planes(g, b):
    """Block Cholesky plane by plane along the longest axis: plane k couples to plane k - 1 by a diagonal matrix."""
    ax = int(np.argmax(g.dims))
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(np.moveaxis(v, ax, 0))).cuda()  # noqa: E731
    diag, edges = dev(g.diag), [dev(e) for e in g.edges]
    link = edges.pop(ax)
    K, m = diag.shape[0], diag[0].numel()
    inner = [d for i, d in enumerate(g.dims) if i != ax]
    cols = np.arange(m).reshape(inner)
    pairs = [(torch.from_numpy(np.take(cols, range(inner[a] - 1), a).reshape(-1)).cuda(),
              torch.from_numpy(np.take(cols, range(1, inner[a]), a).reshape(-1)).cuda()) for a in range(len(inner))]
    diag, link = diag.reshape(K, m), link.reshape(K - 1, m)
    edges = [e.reshape(K, -1) for e in edges]
    nq = b.shape[0]
    B = torch.from_numpy(np.ascontiguousarray(np.moveaxis(b.reshape((nq,) + g.dims), 1 + ax, 0))).cuda()
    B = B.reshape(K, nq, m).transpose(1, 2).contiguous()          # K x m x nq

    def plane(k):
        A = torch.zeros(m, m, dtype=torch.float64, device="cuda")
        A.diagonal().copy_(diag[k])
        for (i, j), e in zip(pairs, edges):
            A[i, j] = -e[k]
            A[j, i] = -e[k]
        return A

    chol = []
    for k in range(K):
        S = plane(k)
        if k:
            W = torch.linalg.solve_triangular(chol[-1], torch.diag(link[k - 1]), upper=False)
            S -= W.T @ W
            del W
        chol.append(torch.linalg.cholesky(S))
        del S

    def solve(R):
        Y, X = [], [None] * K
        for k in range(K):
            r = R[k]
            if k:
                r = r + link[k - 1][:, None] * torch.cholesky_solve(Y[-1], chol[k - 1])
            Y.append(r)
        for k in reversed(range(K)):
            r = Y[k]
            if k + 1 < K:
                r = r + link[k][:, None] * X[k + 1]
            X[k] = torch.cholesky_solve(r, chol[k])
        return torch.stack(X)

    def times(X):
        R = diag[:, :, None] * X
        for (i, j), e in zip(pairs, edges):
            R.index_add_(1, i, -e[:, :, None] * X[:, j])
            R.index_add_(1, j, -e[:, :, None] * X[:, i])
        R[1:] -= link[:, :, None] * X[:-1]
        R[:-1] -= link[:, :, None] * X[1:]
        return R

    X = solve(B)
    X += solve(B - times(X))
    X = X.transpose(1, 2).reshape([K, nq] + inner)
    return torch.movedim(X, 0, 1 + ax).reshape(nq, g.n).contiguous()


def _exact(g, b):
    return _exact_dense(g, b) if g.n <= 6000 else _exact_planes(g, b)


def exact(case, seed):
    if case["kind"] == "batch":
        if case["count"] > 600:
            return None
        grids, bs = _batch_inputs(case, seed)
        return torch.cat([_exact(g, b[None]) for g, b in zip(grids, bs)], 1)
    g, b = _inputs(case, seed)
    x = _exact(g, b)
    return x.T.contiguous() if case["kind"] == "linsolve" else x
