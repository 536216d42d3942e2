"""The coarse operator, bit for bit the oracle's, from rows on both sides of
the kernel's cuts: 8 entries (one pass of a row's threads), 32 (the longest
row staged), rows that touch no other part, one, or many, and a last batch of
listed rows that is not full."""
from __future__ import annotations

import numpy as np
import pytest
from conftest import HostCSR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 3, 7, 8, 9, 16, 17, 32, 33, 40])
@pytest.mark.parametrize("parts", [2, 9, 40])
def test_coarse_operator_bitwise(sg, oracle, width, parts):
    n = 50 * parts + 13
    rng = np.random.default_rng([width, parts])
    cols, vals = [], []
    for i in range(n):
        spread = 3 if rng.random() < 0.4 else n
        k = np.unique(np.append(np.clip(i + rng.integers(-spread, spread + 1, rng.integers(0, width + 1)),
                                        0, n - 1), i))
        cols.append(k)
        v = rng.uniform(-1, 1, k.size)
        v[k == i] = 4.0 * width
        vals.append(v)
    rp = np.cumsum([0] + [c.size for c in cols]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    v = np.concatenate(vals)
    part = (np.arange(n) * parts // n).astype(np.int32)
    M = sg.TwoLevelSchwarzPrecond(parts, 0, sg.FineLevelType.RAS, partition=part)
    M.setup(sg.CSRMatrix(n, n, rp, ci, v))
    ref = oracle.precond("twolevel_ras", HostCSR(rp, ci, v), parts, 0, part).coarse_a0()
    assert np.array_equal(M.coarse_a0(), ref)
