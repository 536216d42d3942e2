"""The blocked LU of the coarse operator at the edges of its panels (16
columns), tiles (32) and of the panels that fit in shared memory (1,690 rows),
on operators whose every column needs a row swap.

Part p couples to part p - 1 two to four times as strongly as to itself, so
A0 = D + S with |D| <= 1.1 and 2 <= |S| <= 4 on the cyclic subdiagonal: its
condition is at most 5.1 / 0.9 < 6, and the two ways to apply its inverse
differ by a few n * 6 * 2^-53 of the result -- 1.2e-12 times the elimination's
growth at n = 1,750, for which 1e-10 leaves two digits.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import HostCSR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 2, 15, 16, 17, 31, 33, 48, 64, 100, 257, 600, 1750])
def test_two_level_apply_with_pivoting(sg, oracle, parts):
    rng = np.random.default_rng(parts)
    n = 2 * parts
    cols, vals = [], []
    for i in range(n):
        e = {i: rng.uniform(0.9, 1.1)}
        j = (i - 2) % n
        if j != i:
            e[j] = e.get(j, 0.0) + rng.uniform(2.0, 4.0) * (1 if rng.random() < 0.5 else -1)
        if i % 2 == 0 and parts > 1:
            # keep a part's two couplings of one sign: they add up in A0
            sign = 1.0 if e[j] > 0 else -1.0
        if i % 2 == 1 and parts > 1:
            e[j] = sign * abs(e[j])
        ks = sorted(e)
        cols.append(ks)
        vals.append([e[k] for k in ks])
    rp = np.cumsum([0] + [len(c) for c in cols]).astype(np.int32)
    ci = np.concatenate([np.array(c, np.int32) for c in cols])
    v = np.concatenate([np.array(c) for c in vals])
    part = (np.arange(n) // 2).astype(np.int32)
    A = sg.CSRMatrix(n, n, rp, ci, v)
    M = sg.TwoLevelSchwarzPrecond(parts, 0, sg.FineLevelType.RAS, partition=part)
    M.setup(A)
    x = rng.standard_normal(n)
    y = M.apply(x)
    ref = oracle.precond("twolevel_ras", HostCSR(rp, ci, v), parts, 0, part).apply(x)
    assert np.max(np.abs(y - ref)) <= 1e-10 * np.max(np.abs(ref))
