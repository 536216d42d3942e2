"""The product with a matrix of uneven rows (which has no SELL copy): bit for
bit the row loop's products and sums at the edges of its blocks of 256 rows
and windows of 4,096 products, with empty rows and rows longer than the
longest length class (63) and than a window; and an FP32 solve with it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uneven(n, longest, seed):
    rng = np.random.default_rng(seed)
    w = np.minimum(rng.geometric(0.15, n), 70)
    w[rng.integers(0, n, n // 5 + 1)] = 0
    w[rng.integers(0, n)] = longest
    rp = np.concatenate([[0], np.cumsum(w)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.integers(0, n, k)) for k in w]).astype(np.int32)
    return w, rp, ci, rng.standard_normal(rp[-1]), rng


@pytest.mark.parametrize("n", [33, 255, 256, 257, 511, 513, 5000])
@pytest.mark.parametrize("longest", [62, 63, 64, 500, 4096, 9001])
def test_uneven_rows_bitwise(sg, n, longest):
    w, rp, ci, v, rng = _uneven(n, longest, n + longest)
    x = rng.standard_normal(n)
    A = sg.CSRMatrix(n, n, rp, ci, v)
    with pytest.raises(sg.SgError):  # no SELL copy: the kernel under test runs
        A.set_spmv_variant(0)
    ref = np.zeros(n)
    for k in range(int(w.max())):
        on = w > k
        e = rp[:-1][on] + k
        ref[on] = ref[on] + v[e] * x[ci[e]]
    assert np.array_equal(A.spmv(x), ref)


def test_uneven_rows_in_an_fp32_solve(sg):
    n = 3000
    w, rp, ci, v, rng = _uneven(n, 300, 5)
    import scipy.sparse as sp

    S = sp.csr_matrix((v, ci, rp), shape=(n, n))
    S = (S + sp.diags(np.abs(S).sum(axis=1).A1 + 1.0)).tocsr()
    S.sort_indices()
    A = sg.CSRMatrix(n, n, S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data)
    b = rng.standard_normal(n)
    x = np.zeros(n)
    M = sg.JacobiPrecond(sweep_dtype=sg.FP32)
    M.setup(A)
    r = sg.gmres(A, b, x, M, sg.GMRESParams(tol=1e-10, tol_kind=sg.TOL_TRUE_REL, precision=sg.FP32))
    assert r.converged
    # the solver's own criterion, recomputed: its FP64 residual rounds n terms
    assert np.linalg.norm(b - S @ x) <= 1.01e-10 * np.linalg.norm(b)
