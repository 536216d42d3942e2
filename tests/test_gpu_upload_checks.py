"""Refusals of an upload: a row_ptr that passes nnz before it decreases is named
by the row where it decreases, and no column beyond nnz is looked at."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rp,row", [([0, 1000, 5], 1), ([0, 2, 900, 800, 5], 2), ([0, 7, 5], 1)])
def test_row_ptr_beyond_nnz(sg, rp, row):
    A = sg.CSRMatrix(len(rp) - 1, 8, np.array(rp, np.int32), np.arange(5, dtype=np.int32), np.ones(5))
    with pytest.raises(sg.SgError, match=f"row_ptr decreases at row {row}"):
        A.upload()


def test_bad_column_before_the_decrease(sg):
    A = sg.CSRMatrix(3, 8, np.array([0, 2, 900, 5], np.int32), np.array([0, 9, 1, 2, 3], np.int32), np.ones(5))
    with pytest.raises(sg.SgError, match=r"col_idx\[1\] = 9 outside \[0,8\)"):
        A.upload()


@pytest.mark.parametrize("n", [2, 40, 1000])
def test_sorted_rows_are_told_by_entry(sg, n):
    """Only a decrease inside a row makes it unsorted (no SELL copy): not the
    one from row to row, with empty rows between or none; and a column out of
    range is named wherever it is."""
    i = np.arange(n)
    ci = np.stack([i * 0, i * 0 + n // 2, i * 0 + n - 1], 1)[:, :2 if n < 3 else 3].astype(np.int32)
    w = ci.shape[1]
    v = np.ones(ci.size)
    for rp in (w * np.arange(n + 1), np.append(0, w * np.arange(1, n + 1))):
        A = sg.CSRMatrix(n, n, rp.astype(np.int32), ci.ravel().copy(), v)
        A.upload()
        A.format = 2
    for k in {0, n // 2, n - 1}:
        bad = ci.copy()
        bad[k] = bad[k][::-1]
        if n > 2 or k == 0:
            A = sg.CSRMatrix(n, n, (w * np.arange(n + 1)).astype(np.int32), bad.ravel(), v)
            A.upload()
            with pytest.raises(sg.SgError, match="no SELL copy"):
                A.format = 2
        far = ci.copy()
        far[k, w - 1] = n
        with pytest.raises(sg.SgError, match=rf"col_idx\[{k * w + w - 1}\] = {n} outside"):
            sg.CSRMatrix(n, n, (w * np.arange(n + 1)).astype(np.int32), far.ravel(), v).upload()
    # rows of one and two entries with empty rows between
    rows = np.where(i % 3 == 0, 0, 1 + i % 2)
    rp = np.concatenate([[0], np.cumsum(rows)]).astype(np.int32)
    cc = np.concatenate([np.arange(k, dtype=np.int32) for k in rows])
    sg.CSRMatrix(n, n, rp, cc, np.ones(cc.size)).upload()


def test_upload_of_a_long_row(sg):
    """A matrix with a row of 3 million entries is uploaded in about the time of
    as many entries in short rows (the copies' time; with its entries checked one
    after another it took 50 times that)."""
    import time

    n = 50000
    long, even = np.full(n, 5), np.full(n, 65)
    long[n // 2] = 3_000_000
    runs = []
    for w in (even, long):
        rp = np.concatenate([[0], np.cumsum(w)]).astype(np.int32)
        runs.append((sg.CSRMatrix(n, n, rp, np.zeros(rp[-1], np.int32), np.ones(rp[-1])), []))
    for _ in range(5):
        for A, s in runs:
            t = time.perf_counter()
            A.upload()
            s.append(time.perf_counter() - t)
    assert min(runs[1][1]) < 8 * min(runs[0][1])
