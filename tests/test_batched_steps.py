"""Batched restart cycles whose steps cross the pass kernels' sizes (4, 8, ...
32 vectors held by a thread), with systems from one row to several chunks of
2,048 rows, one to five right-hand sides and both forms of CGS2: every
solution against a dense solve of its system."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(sg, sizes, seed):
    """Block-diagonal union of random diagonally dominant banded systems."""
    r = np.random.default_rng(seed)
    rp, ci, v, rows, dense = [0], [], [], [0], []
    for n in sizes:
        a = np.zeros((n, n))
        for d in (1, 2, 7):
            if n > d:
                a += np.diag(r.uniform(-1, 1, n - d), d) + np.diag(r.uniform(-1, 1, n - d), -d)
        a += np.diag(np.abs(a).sum(1) + 0.05)
        dense.append(a)
        for i in range(n):
            c = np.flatnonzero(a[i])
            ci.extend(c + rows[-1])
            v.extend(a[i, c])
            rp.append(len(ci))
        rows.append(rows[-1] + n)
    A = sg.CSRMatrix(rows[-1], rows[-1], np.array(rp, np.int32), np.array(ci, np.int32), np.array(v))
    return A, np.array(rows, np.int32), dense


@pytest.mark.parametrize("restart", [1, 4, 5, 9, 16, 24, 28, 31, 32])
@pytest.mark.parametrize("nrhs", [1, 4, 5])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_every_step_size(sg, restart, nrhs, precision):
    sizes = [1, 2, 31, 257, 2049] if restart == 31 else [1, 33, 200]
    A, rows, dense = _batch(sg, sizes, restart)
    n = A.nrows
    B = sg.uniform(nrhs * n, seed=restart).reshape(nrhs, n)
    X = np.zeros_like(B)
    M = sg.JacobiPrecond()
    M.setup(A)
    res, _ = sg.solve_batched(A, M, rows, nrhs, B, X, sg.GMRESParams(
        restart=restart, max_iter=4000, tol=1e-10, tol_kind=sg.TOL_TRUE_REL,
        precision=sg.FP64 if precision == "fp64" else sg.FP32))
    assert np.all(res["converged"] == 1)
    for s, a in enumerate(dense):
        for r in range(nrhs):
            b, x = B[r, rows[s]: rows[s + 1]], X[r, rows[s]: rows[s + 1]]
            # the solver's own criterion, rounding of the check added
            assert np.linalg.norm(b - a @ x) <= 1.0001e-10 * np.linalg.norm(b)
