"""The batched solver keeps its tables between solves of one matrix.  A matrix
uploaded again -- often to the address of the one before -- is checked again: a
pattern of the same size that couples two systems is refused."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_new_pattern_is_checked_again(sg):
    n = 400
    i = np.arange(n)
    rp = (2 * np.arange(n + 1)).astype(np.int32)
    own = np.sort(np.stack([i, i ^ 1], 1), 1).ravel().astype(np.int32)  # systems of two rows
    far = own.copy()
    far[1] = 20  # row 0: its neighbour is in another system
    v = np.where(own == np.repeat(i, 2), 4.0, 1.0)
    rows = np.arange(0, n + 1, 2, dtype=np.int32)
    b = sg.uniform(n, 1).reshape(1, n)

    def solve(A, M):
        M.setup(A)
        x = np.zeros((1, n))
        return sg.solve_batched(A, M, rows, 1, b, x, sg.GMRESParams(
            restart=2, max_iter=4000, tol=1e-12, tol_kind=sg.TOL_TRUE_REL))[0]

    for _ in range(40):  # the address is the same in about a third of them
        ctx = sg.Context(0)
        M = sg.JacobiPrecond(ctx=ctx)
        for _ in range(2):
            A = sg.CSRMatrix(n, n, rp, own, v)
            A.upload(ctx)
            assert np.all(solve(A, M)["converged"] == 1)
        A.col_idx = far
        A.upload(ctx)
        with pytest.raises(sg.SgError, match="row 0 couples system 0 to column 20"):
            solve(A, M)
