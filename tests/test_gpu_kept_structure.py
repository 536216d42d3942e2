"""A set-up with new values of the same structure keeps the structure's arrays
and plans on the device; what it computes is what a new preconditioner set up
with those values computes, bit for bit -- also after a set-up of another
structure and back, and after one that failed on its values."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = [("ilu0", "FP64", 1), ("ras", "FP64", 8), ("ras", "FP32", 8), ("asm", "FP32", 8),
         ("twolevel_ras", "FP64", 8), ("twolevel_ras", "BF16", 8), ("twolevel_asm", "FP32", 8)]


def _make(sg, kind, dt, parts, n):
    fd = getattr(sg, dt)
    sd = sg.FP64 if dt == "FP64" else sg.FP32
    if kind == "ilu0":
        return sg.ILU0Precond(fd, sd)
    part = np.arange(n, dtype=np.int32) * parts // n
    if kind == "ras":
        return sg.RASPrecond(parts, 1, part, fd, sd)
    if kind == "asm":
        return sg.ASMPrecond(parts, 1, part, fd, sd)
    lvl = sg.FineLevelType.RAS if kind == "twolevel_ras" else sg.FineLevelType.ASM
    return sg.TwoLevelSchwarzPrecond(parts, 1, lvl, part, fd, sd)


@pytest.mark.parametrize("kind,dt,parts", KINDS)
def test_new_values_match_a_new_preconditioner(sg, kind, dt, parts):
    N = 16
    A = sg.make_varcoef_3d(N, N, N, 1.0, 3.0, 1)
    vals = [sg.make_varcoef_3d(N, N, N, 1.0, 3.0, s).vals.copy() for s in (1, 2, 3)]
    other = sg.make_varcoef_3d(N, N, 2 * N, 1.0, 3.0, 4)  # another structure
    x = np.random.default_rng(0).standard_normal(A.nrows)
    M = _make(sg, kind, dt, parts, A.nrows)
    M.setup(A)

    def check(v):
        A.vals = v
        A.upload()
        M.setup(A)
        F = _make(sg, kind, dt, parts, A.nrows)
        F.setup(A)
        a, b = M.apply(x), F.apply(x)
        if "asm" in kind:  # overlapping rows are added atomically, in any order
            # a row is owned by one part and in at most all 8 overlaps: 8 terms
            # and the coarse one, each addition rounded in FP64
            assert np.max(np.abs(a - b)) <= 9 * 2.0 ** -53 * 9 * np.max(np.abs(b))
        else:
            assert np.array_equal(a, b)

    check(vals[1])
    if kind == "ilu0":
        M.setup(other)
        check(vals[2])
    A.vals = np.zeros_like(vals[0])  # singular: the set-up fails or its result is not finite
    A.upload()
    try:
        M.setup(A)
    except sg.SgError:
        pass
    check(vals[0])
