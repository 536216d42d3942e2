"""The dot products of the batched FP32 basis are summed over the rows in FP64
(each product in FP32, its sum over threads not)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cancelling_dot_keeps_53_bits(sg):
    """One step from b with 16 ones (beta = 4) on a diagonal matrix: v . A v =
    2^-4 (1 + 2^-24 + 2^-48 - 1 - 2^-24).  Every partial sum, in any order, has
    at most 53 bits, and so has every one of the second projection's, after the
    update by u = 2^-54 that FP32 rounds away in the large rows: h = 2^-52 +
    2^-54, ||w||^2 = 2 (1/4)^2 and a few 2^-52, and the step's solution is
    h / ||w||^2 = 10 * 2^-52 in the rows with ones.  Sums of fewer bits give 0.
    Tolerance: the coefficient is rounded to FP32 (2^-24), ||w||^2 to 2^-49."""
    n = 32
    d = np.zeros(n)
    d[[0, 16, 8, 4, 2]] = 1.0, 2.0 ** -24, 2.0 ** -48, -1.0, -(2.0 ** -24)
    b = np.zeros((1, n))
    b[0, [0, 16, 8, 4, 2]] = 1.0
    b[0, [1, 3, 5, 6, 7, 9, 10, 11, 12, 13, 14]] = 1.0
    i = np.arange(n, dtype=np.int32)
    A = sg.CSRMatrix(n, n, np.arange(n + 1, dtype=np.int32), i, d)
    x = np.zeros((1, n))
    sg.solve_batched(A, None, np.array([0, n], np.int32), 1, b, x, sg.GMRESParams(
        restart=1, max_iter=1, tol=1e-12, tol_kind=sg.TOL_TRUE_REL, precision=sg.FP32))
    assert np.allclose(x, 10 * 2.0 ** -52 * b, rtol=2.0 ** -23, atol=0.0)


def test_product_scaled_in_fp64(sg):
    """w = A v is the FP32 product times 1 / ||raw|| in FP64, rounded once.  One
    step of one-row systems a x = b whose w lies next to a midpoint of two
    floats, restated: x = fl32(fl32(y / beta) b), y = beta / h."""
    f = np.float32
    ab = [("0x1.43348ap+0", "0x1.1d21eap+0"), ("0x1.1129c8p+0", "0x1.7a827ep+0"),
          ("0x1.7f236ep+0", "0x1.4ea5a4p+0"), ("0x1.96a474p+0", "0x1.aef49ep+0"),
          ("0x1.96a476p+0", "0x1.aef49ep+0")]
    a = np.array([float.fromhex(s) for s, _ in ab])
    b = np.array([float.fromhex(s) for _, s in ab])
    want = []
    for ai, bi in zip(a, b):
        raw = f(bi)
        beta = float(np.sqrt(float(f(raw * raw))))
        T = 1.0 / beta
        z = f(float(f(f(ai) * raw)) * T)
        p = T * float(f(raw * z))
        w = f(float(z) - float(f(T * p)) * float(raw))  # one rounding: exact in FP64
        h2 = T * float(f(raw * w))
        h = p + h2
        assert float(f(w * w)) - h2 * h2 > 0.0  # no breakdown, which would start another cycle
        want.append(float(f(f(beta / h * T) * raw)))
    n = len(ab)
    x = np.zeros((1, n))
    sg.solve_batched(sg.CSRMatrix(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), a),
                     None, np.arange(n + 1, dtype=np.int32), 1, b.reshape(1, n), x, sg.GMRESParams(
                         restart=1, max_iter=1, tol=1e-14, tol_kind=sg.TOL_TRUE_REL, precision=sg.FP32))
    assert np.array_equal(x[0], np.array(want))
