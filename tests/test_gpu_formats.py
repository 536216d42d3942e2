"""The SELL-32 copy, its 16-bit column offsets and the FP32 values are made on
the device: every format of a matrix gives the bits of the row-by-row CSR
product, at sizes around a slice's 32 rows, with empty rows, with rows too
uneven to keep the copy, with columns too far for 16 bits, and unsorted."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(sg, n, widths, reach, seed, sort=True):
    r = np.random.default_rng(seed)
    cols = []
    for i, w in enumerate(widths):
        lo, hi = max(0, i - reach), min(n, i + reach + 1)
        c = r.choice(np.arange(lo, hi), size=min(w, hi - lo), replace=False)
        cols.append(np.sort(c) if sort else c)
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    return sg.CSRMatrix(n, n, rp, ci, r.standard_normal(ci.size))


def _reference(A, x):
    y = np.zeros(A.nrows)
    for i in range(A.nrows):
        for e in range(A.row_ptr[i], A.row_ptr[i + 1]):
            y[i] += A.vals[e] * x[A.col_idx[e]]
    return y


@pytest.mark.parametrize("n", [1, 31, 32, 33, 95, 4097])
@pytest.mark.parametrize("kind", ["even", "holes", "uneven"])
def test_formats_agree(sg, n, kind):
    r = np.random.default_rng(n)
    w = np.full(n, 5)
    if kind == "holes":
        w = r.integers(4, 6, n)
        w[r.random(n) < 0.05] = 0
    elif kind == "uneven":
        w = np.where(r.random(n) < 0.03, 60, 2)
    A = _csr(sg, n, w, 40, n)
    x = sg.uniform(n, 3)
    want = _reference(A, x)
    rows = np.diff(A.row_ptr)
    entries = sum(32 * int(rows[s: s + 32].max()) for s in range(0, n, 32))
    kept = entries <= A.nnz() + A.nnz() // 4 + 64  # the copy's padding bound
    for fmt in (0, 1, 2, 3):
        if fmt >= 2 and not kept:
            with pytest.raises(sg.SgError):
                A.format = fmt
            continue
        A.format = fmt
        assert np.array_equal(A.spmv(x), want), fmt


def test_far_columns_have_no_short_offsets(sg):
    n = 40000
    i = np.arange(n)
    far = (i + 33000) % n
    lo, hi = np.minimum(i, far), np.maximum(i, far)
    ci = np.stack([lo, hi], 1).reshape(-1).astype(np.int32)
    A = sg.CSRMatrix(n, n, np.arange(0, 2 * n + 1, 2, dtype=np.int32), ci, sg.uniform(2 * n, 5))
    x = sg.uniform(n, 6)
    A.format = 1
    want = A.spmv(x)
    A.format = 2
    assert np.array_equal(A.spmv(x), want)
    with pytest.raises(sg.SgError):
        A.format = 3


def test_unsorted_rows_stay_csr(sg):
    A = _csr(sg, 200, np.full(200, 6), 50, 9, sort=False)
    x = sg.uniform(200, 7)
    assert np.array_equal(A.spmv(x), _reference(A, x))
    with pytest.raises(sg.SgError):
        A.format = 2


def test_bad_columns_are_refused_by_name(sg):
    A = _csr(sg, 100, np.full(100, 4), 20, 1)
    A.col_idx[37] = 100
    with pytest.raises(sg.SgError, match=r"col_idx\[37\] = 100"):
        A.upload()
    A.col_idx[37] = -1
    with pytest.raises(sg.SgError, match=r"col_idx\[37\] = -1"):
        A.upload()
