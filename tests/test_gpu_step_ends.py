"""The end of an Arnoldi step rounds as the reference's formulas do
(src/core/gmres.cpp:9-30): the norm is a correctly rounded root, the rotation
1 / sqrt(1 + t^2) a root and a quotient.  From b = e_1 and integer columns
(p, q) every dot product and ||w''||^2 = q^2 is exact, so the first residual is
known to the last bit."""
from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _residual(p, q):
    t = -(p / q) if q > p else -(q / p)
    r = 1.0 / np.sqrt(float(1 + Fraction(t) ** 2))  # one rounding: a fused multiply-add
    return abs(r if q > p else r * t)


@pytest.mark.parametrize("restart", [5, 40])
def test_first_residual_to_the_last_bit(sg, restart):
    rng = np.random.default_rng(restart)
    b = np.array([1.0, 0.0])
    rp, ci = np.array([0, 1, 3], np.int32), np.array([0, 0, 1], np.int32)
    got, want = [], []
    for _ in range(200):
        p, q = (int(v) for v in rng.integers(1, 1 << 26, 2))
        A = sg.CSRMatrix(2, 2, rp, ci, np.array([p, q, 3.0]))
        r = sg.gmres(A, b, np.zeros(2), None, sg.GMRESParams(restart=restart, max_iter=1, tol=1e-300))
        got.append(r.residual_history[0])
        want.append(_residual(float(p), float(q)))
    assert np.array_equal(got, want)
