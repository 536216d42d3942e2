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
