"""A dot product of the FP32 basis sums the four products of a 16-byte load
before it adds them to the running sum."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_products_of_a_load_are_summed_first(sg):
    """One step from b with 16 ones (beta = 4) on a diagonal matrix, in 128
    tiles of 128 rows.  A lane of the first tile group adds 2^25 from tile 0 and
    1 + 1 + 1 + 1 from one load of tile 64, its neighbour -2^25; the other ten
    ones meet zeros, each in a warp of its own.  v . A v is 4 / 4 = 1; the
    update by 1/4 rounds away in the large rows and leaves 3/4 in the four and
    -1/4 in the ten, whose second dot is (2^25 + 3 = 2^25 + 4 in FP32) 4 - 2.5,
    over 4 again: h = 1.375, ||w||^2 = 2^51 (1 + 2^-48), and the step's solution
    is h 2^-51 in the rows with ones, its coefficient rounded to FP32 (2^-24).
    Added one by one, the fours are lost."""
    n = 128 * 128
    d, b = np.zeros(n), np.zeros(n)
    d[[0, 4]] = 2.0 ** 27, -(2.0 ** 27)
    d[64 * 128: 64 * 128 + 4] = 4.0
    b[d != 0] = 1.0
    b[128 * np.arange(1, 11)] = 1.0
    A = sg.CSRMatrix(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d)
    x = np.zeros(n)
    sg.gmres(A, b, x, None, sg.GMRESParams(restart=1, max_iter=1, tol=1e-12, precision=sg.FP32,
                                          tol_kind=sg.TOL_TRUE_REL))
    assert np.allclose(x, 1.375 * 2.0 ** -51 * b, rtol=2.0 ** -23, atol=0.0)
