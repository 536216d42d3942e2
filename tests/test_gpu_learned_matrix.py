"""The learned stage reads its matrix's diagonal on the device: entries of one
place are added in their order, wherever they stand in the row, and a row whose
diagonal is not positive is named."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 16


def _feature(sg, A, M):
    st = sg.LearnedCorrection(N)
    try:
        st.set_matrix(A)
        st.add_pair(M, sg.uniform(A.nrows, 1), sg.uniform(A.nrows, 2))
        return st.sample(0)[1]
    finally:
        st.close()


def test_diagonal_in_parts(sg):
    A = sg.make_varcoef_3d(N, N, N, 1.0, 3.0, 1)
    n = A.nrows
    rng = np.random.default_rng(3)
    one, rows = A.vals.copy(), []
    for i in range(n):
        s = slice(A.row_ptr[i], A.row_ptr[i + 1])
        c, v = A.col_idx[s], A.vals[s]
        k = int(np.flatnonzero(c == i)[0])
        if i % 5 == 0:  # three parts, the last behind up to 70 zeros
            z = int(rng.integers(0, 70))
            p = v[k] * np.array([0.3, 0.45, 0.25])
            one[A.row_ptr[i] + k] = (0.0 + p[0] + p[1]) + p[2]
            c = np.concatenate([c[:k], [i, i], c[k + 1:], np.full(z, (i + 1) % n), [i]])
            v = np.concatenate([v[:k], p[:2], v[k + 1:], np.zeros(z), p[2:]])
        rows.append((c, v))
    rp = np.concatenate([[0], np.cumsum([c.size for c, _ in rows])]).astype(np.int32)
    B = sg.CSRMatrix(n, n, rp, np.concatenate([c for c, _ in rows]).astype(np.int32),
                     np.concatenate([v for _, v in rows]))
    C = sg.CSRMatrix(n, n, A.row_ptr, A.col_idx, one)
    M = sg.JacobiPrecond()
    M.setup(C)
    f = _feature(sg, B, M)
    assert np.array_equal(f, _feature(sg, C, M)) and np.std(f) > 0.5


@pytest.mark.parametrize("row", [0, 77, N ** 3 - 1])
@pytest.mark.parametrize("value", [0.0, -1.0, np.nan])
def test_diagonal_not_positive(sg, row, value):
    A = sg.make_varcoef_3d(N, N, N, 1.0, 3.0, 1)
    v = A.vals.copy()
    v[A.row_ptr[row] + np.flatnonzero(A.col_idx[A.row_ptr[row]: A.row_ptr[row + 1]] == row)[0]] = value
    st = sg.LearnedCorrection(N)
    with pytest.raises(sg.SgError, match=f"row {row} has a non-positive diagonal"):
        st.set_matrix(sg.CSRMatrix(A.nrows, A.nrows, A.row_ptr, A.col_idx, v))
    st.close()
