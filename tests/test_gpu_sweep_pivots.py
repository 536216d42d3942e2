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
