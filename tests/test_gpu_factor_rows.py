"""ILU(0) factors bit for bit against the oracle where the factorisation's two
ways to take a row meet: rows of up to 9 entries with up to 4 pivots whose
rows hold up to 4 entries above the diagonal, and anything beyond, mixed in
one matrix; zero and tiny pivots; non-finite values; and the refusal of a missing pivot."""
from __future__ import annotations

import numpy as np
import pytest
from conftest import HostCSR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [1, 2, 3, 4, 5, 7])
@pytest.mark.parametrize("odd", ["none", "pivots", "nonfinite", "tiny"])
def test_factors_bitwise(sg, oracle, half, odd):
    n = 700
    rng = np.random.default_rng(half)
    cols, vals = [], []
    for i in range(n):
        near = i + rng.integers(-20, 21, size=rng.integers(0, half + 1))
        far = rng.integers(0, n, size=rng.integers(0, half + 1))
        k = np.unique(np.concatenate([near[(near >= 0) & (near < n)], far, [i]]))
        if odd == "pivots" and rng.random() < 0.1:
            k = k[k != i] if k.size > 1 else k
        v = rng.uniform(-1, 1, k.size)
        v[k == i] = rng.uniform(2, 4) * half
        if odd in ("pivots", "tiny") and rng.random() < 0.1:
            v[k == i] = rng.choice([0.0, -0.0, 1e-31, -9e-31, 5e-324, 1.1e-30])
        if odd == "nonfinite" and rng.random() < 0.01:
            v[rng.integers(0, k.size)] = rng.choice([np.inf, -np.inf, np.nan])
        cols.append(k)
        vals.append(v)
    rp = np.cumsum([0] + [c.size for c in cols]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    v = np.concatenate(vals)
    part = (np.arange(n) * 3 // n).astype(np.int32)
    M = sg.RASPrecond(3, 1, part)
    A = sg.CSRMatrix(n, n, rp, ci, v)
    if odd == "pivots":  # a row without a diagonal entry is refused
        with pytest.raises(sg.SgError, match="no diagonal entry"):
            M.setup(A)
        return
    M.setup(A)
    po = oracle.precond("ras", HostCSR(rp, ci, v), 3, 1, part)
    for s in range(3):
        _, oc, lu, _ = po.sub_factor(s)
        f = M.factors(s)
        assert np.array_equal(f["col_idx"], oc)
        a, b = np.asarray(f["lu_vals"]), np.asarray(lu)
        assert np.array_equal(np.isnan(a), np.isnan(b))
        ok = ~np.isnan(b)
        assert np.array_equal(a[ok].view(np.uint64), b[ok].view(np.uint64))
