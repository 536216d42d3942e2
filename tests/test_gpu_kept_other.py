"""Between set-ups of one structure, a partitioned preconditioner set up with
another pattern of the same rows and partition, or refused on one, computes
afterwards what a new preconditioner computes, bit for bit; and a batch of four
right-hand sides keeps its plan over a set-up with new values."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, PARTS = 48, 8
KINDS = [("ras", "FP64"), ("ras", "FP32"), ("ras", "BF16"), ("asm", "FP64"),
         ("twolevel_ras", "FP64"), ("twolevel_ras", "BF16"), ("twolevel_asm", "FP32")]


def _make(sg, kind, dt, part):
    fd, sd = getattr(sg, dt), sg.FP64 if dt == "FP64" else sg.FP32
    if kind == "ras":
        return sg.RASPrecond(PARTS, 1, part, fd, sd)
    if kind == "asm":
        return sg.ASMPrecond(PARTS, 1, part, fd, sd)
    lvl = sg.FineLevelType.RAS if kind == "twolevel_ras" else sg.FineLevelType.ASM
    return sg.TwoLevelSchwarzPrecond(PARTS, 1, lvl, part, fd, sd)


@pytest.mark.parametrize("kind,dt", KINDS)
def test_another_pattern_and_back(sg, kind, dt):
    five, nine = sg.make_poisson_2d(N, N), sg.make_aniso_2d(N, N, 0.3, 0.6)
    n = five.nrows
    part = sg.partition_boxes(N, N, 1, PARTS, 0.1, seed=3)
    x = np.random.default_rng(0).standard_normal(n)
    M = _make(sg, kind, dt, part)

    def check(A):
        M.setup(A)
        F = _make(sg, kind, dt, part)
        F.setup(A)
        assert M.check() == 0
        a, b = M.apply(x), F.apply(x)
        if "asm" in kind:  # overlapping rows are added atomically: at most 9 terms, any order
            assert np.max(np.abs(a - b)) <= 9 * 2.0 ** -53 * 9 * np.max(np.abs(b))
        else:
            assert np.array_equal(a, b)

    wide = sg.CSRMatrix(n, n, five.row_ptr, five.col_idx, five.vals * np.where(five.vals > 0, 1.5, 1.0))
    for A in (five, wide, nine, five, wide):
        check(A)
    # a row without a diagonal entry is refused
    k = int(np.flatnonzero(five.col_idx[five.row_ptr[7]: five.row_ptr[8]] == 7)[0] + five.row_ptr[7])
    rp = five.row_ptr.copy()
    rp[8:] -= 1
    with pytest.raises(sg.SgError, match="no diagonal entry"):
        M.setup(sg.CSRMatrix(n, n, rp, np.delete(five.col_idx, k), np.delete(five.vals, k)))
    check(wide)
    if kind.startswith("twolevel"):
        with pytest.raises(sg.SgError):  # a coarse operator of zeros
            M.setup(sg.CSRMatrix(n, n, five.row_ptr, five.col_idx, 0.0 * five.vals))
        check(five)
        check(nine)


@pytest.mark.parametrize("dt", ["FP32", "BF16"])
def test_four_right_hand_sides_after_new_values(sg, dt):
    A = sg.make_aniso_2d(N, N, 0.3, 0.6)
    n = A.nrows
    part = sg.partition_boxes(N, N, 1, PARTS, 0.1, seed=3)
    B = sg.uniform(4 * n, 2).reshape(4, n)
    M = sg.RASPrecond(PARTS, 1, part, getattr(sg, dt), sg.FP32)

    def solve(P):
        P.setup(A)
        X = np.zeros((4, n))
        r = sg.solve_batched(A, P, np.array([0, n], np.int32), 4, B, X, sg.GMRESParams(
            restart=20, max_iter=200, tol=1e-8, tol_kind=sg.TOL_TRUE_REL, precision=sg.FP32))[0]
        assert np.all(r["converged"] == 1)
        return X

    for scale in (1.0, 1.3, 0.8):  # the second and third keep the structure
        A.vals = A.vals * np.where(A.vals > 0, scale, 1.0)
        A.upload()
        assert np.array_equal(solve(M), solve(sg.RASPrecond(PARTS, 1, part, getattr(sg, dt), sg.FP32)))
