"""Sweeps over rows whose pivots are so small that their reciprocal overflows
(|d| < 2^-1024), against the division: FP64 applies equal the oracle bit for
bit, zeros of both signs over such pivots among them."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TINY = [5e-324, 1e-310, -3e-309, 2.0 ** -1024, 2.0 ** -1023, 1e-300]


def _blocks(sg, width, nblk=9, m=7):
    """Disconnected m x m grids (rows of `width` entries a triangle); in every
    third one the diagonals of some rows are tiny.  Returns the matrix and the
    rows of those grids."""
    if width == 2:
        G = sg.make_poisson_2d(m, m)
    elif width == 3:
        G = sg.make_varcoef_3d(m, m, 2, 1.0, 3.0, 1)
    else:
        G = sg.make_aniso_2d(m, m, 0.3, 0.6)
    n = G.nrows
    rp = np.concatenate([[0]] + [np.asarray(G.row_ptr[1:]) + b * G.row_ptr[-1] for b in range(nblk)])
    ci = np.concatenate([np.asarray(G.col_idx) + b * n for b in range(nblk)])
    v = np.tile(np.asarray(G.vals), nblk)
    row = np.repeat(np.arange(nblk * n), np.diff(rp))
    rng = np.random.default_rng(width)
    small = (row // n) % 3 == 1
    d = np.flatnonzero((row == ci) & small)
    d = d[rng.random(d.size) < 0.4]
    v[d] = rng.choice(TINY, d.size)
    A = sg.CSRMatrix(nblk * n, nblk * n, rp.astype(np.int32), ci.astype(np.int32), v)
    return A, np.flatnonzero((np.arange(nblk * n) // n) % 3 == 1)


@pytest.mark.parametrize("width", [2, 3, 4])
@pytest.mark.parametrize("threads", [0, 64, 256])
def test_zeros_over_tiny_pivots(sg, oracle, width, threads):
    A, rows = _blocks(sg, width)
    x = sg.uniform(A.nrows, 3) - 0.5
    x[rows] = np.where(np.arange(rows.size) % 2, 0.0, -0.0)
    part = np.zeros(A.nrows, np.int32)
    part[A.nrows // 2:] = 1
    M = sg.RASPrecond(2, 0, part, sweep_threads=threads)
    M.setup(A)
    assert M.sweep_choice()["sweep"] == "tma" and M.check() == 0
    y = M.apply(x)
    ref = oracle.precond("ras", A, 2, 0, part).apply(x)
    assert np.all(np.isfinite(ref))
    assert np.array_equal(y.view(np.uint64), np.asarray(ref).view(np.uint64))


def _matrix(sg, width):
    if width == 2:
        return sg.make_poisson_2d(40, 33), (40, 33, 1)
    if width == 3:
        return sg.make_varcoef_3d(13, 11, 9, 1.0, 3.0, 1), (13, 11, 9)
    return sg.make_aniso_2d(31, 37, 0.3, 0.6), (31, 37, 1)


def _solve(sg, A, M, b, precision):
    M.setup(A)
    x = np.zeros(A.nrows)
    r = sg.gmres(A, b, x, M, sg.GMRESParams(restart=20, max_iter=60, tol=1e-11, precision=precision,
                                            tol_kind=sg.TOL_TRUE_REL))
    return x, np.array(r.residual_history), r


@pytest.mark.parametrize("width", [2, 3, 4])
@pytest.mark.parametrize("threads", [0, 64, 256])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_solver_sweeps_divide(sg, width, threads, precision):
    """The FP64 sweeps of a solve against those that divide row by row (the
    sync-free ones): the same residual history and solution, bit for bit."""
    A, g = _matrix(sg, width)
    part = sg.partition_boxes(*g, 4, 0.1, seed=2)
    b = sg.uniform(A.nrows, 5) - 0.5
    p = sg.FP64 if precision == "fp64" else sg.FP32
    M = sg.RASPrecond(4, 1, part, sweep_threads=threads)
    x, h, _ = _solve(sg, A, M, b, p)
    assert M.sweep_choice()["sweep"] == "tma"
    y, k, _ = _solve(sg, A, sg.RASPrecond(4, 1, part, sweep="syncfree"), b, p)
    assert np.array_equal(h, k) and np.array_equal(x, y)


@pytest.mark.parametrize("width", [2, 3, 4])
def test_solve_with_tiny_pivots(sg, width):
    """Pivots whose reciprocal overflows in systems whose right-hand side is
    zero: the solve converges as it does when the sweeps divide; a set-up with
    ordinary values after it, and back, computes what a new one does."""
    A, rows = _blocks(sg, width)
    part = (np.arange(A.nrows) * 2 // A.nrows).astype(np.int32)
    b = sg.uniform(A.nrows, 5) - 0.5
    b[rows] = 0.0
    M = sg.RASPrecond(2, 0, part)
    x, h, r = _solve(sg, A, M, b, sg.FP64)
    assert r.converged and M.check() == 0 and M.sweep_choice()["sweep"] == "tma"
    y, k, _ = _solve(sg, A, sg.RASPrecond(2, 0, part, sweep="syncfree"), b, sg.FP64)
    assert np.array_equal(h, k) and np.array_equal(x, y)
    tiny, v = A.vals, A.vals.copy()
    v[np.abs(v) < 1e-200] = 4.0
    for vals in (v, tiny):
        A.vals = vals
        A.upload()
        x, h, _ = _solve(sg, A, M, b, sg.FP64)
        y, k, _ = _solve(sg, A, sg.RASPrecond(2, 0, part), b, sg.FP64)
        assert M.check() == 0 and np.array_equal(h, k) and np.array_equal(x, y)
