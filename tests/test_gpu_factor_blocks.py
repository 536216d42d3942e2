"""ILU(0) factors bit for bit against the oracle for both block sizes of the
factorisation: subdomains that have an SM each and more of them than SMs, with
levels of fewer, as many and more rows than a block has threads."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 2, 151, 152, 153, 400])
def test_factors_bitwise(sg, oracle, parts):
    A = sg.make_poisson_2d(560, 560) if parts < 3 else sg.make_aniso_2d(90, 110, 0.3, 0.6)
    A.vals = A.vals * (1.0 + 0.1 * sg.uniform(A.vals.size, 3))
    part = (np.arange(A.nrows) * parts // A.nrows).astype(np.int32)
    M = sg.RASPrecond(parts, 1, part)
    M.setup(A)
    po = oracle.precond("ras", A, parts, 1, part)
    for s in sorted({0, parts // 2, parts - 1}):
        _, oc, lu, _ = po.sub_factor(s)
        f = M.factors(s)
        assert np.array_equal(f["col_idx"], oc)
        assert np.array_equal(np.asarray(f["lu_vals"]).view(np.uint64), np.asarray(lu).view(np.uint64))
