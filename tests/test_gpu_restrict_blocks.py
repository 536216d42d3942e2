"""The coarse restriction inside the sweep, with blocks of its own (few
subdomains), with blocks that take up to four each (about the number of SMs)
and in the sweeping blocks (more): the bits of the kernel that computes it
alone, on every apply of a sequence (the counters start over)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("parts", [1, 2, 3, 31, 75, 76, 77, 121, 122, 123, 151, 152, 153, 250, 304])
@pytest.mark.parametrize("dt", ["FP64", "BF16"])
def test_restriction_in_the_sweep(sg, parts, dt):
    A = sg.make_poisson_2d(67, 59)
    part = (np.arange(A.nrows, dtype=np.int64) * parts // A.nrows).astype(np.int32)
    fd = getattr(sg, dt)
    sd = sg.FP64 if dt == "FP64" else sg.FP32
    M, F = (sg.TwoLevelSchwarzPrecond(parts, 1, sg.FineLevelType.RAS, part, fd, sd, fuse_restrict=f)
            for f in (True, False))
    M.setup(A)
    F.setup(A)
    rng = np.random.default_rng(parts)
    for _ in range(4):
        x = rng.standard_normal(A.nrows)
        assert np.array_equal(M.apply(x), F.apply(x))
