"""The product with rows so long that a warp takes 32 of them by itself, in a
block of 256 rows beside blocks that deal their rows by length: bit for bit the
row loop, with rows around the line between the two ways, non-square, unsorted;
and no slower than the rows' own warps are."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 256, 300, 1000])
@pytest.mark.parametrize("kind", ["even", "around", "some", "one"])
def test_long_rows_bitwise(sg, n, kind):
    rng = np.random.default_rng(n)
    w = np.minimum(rng.geometric(0.2, n), 60)
    if kind == "even":
        w[:] = 1500
    elif kind == "around":  # rows of 600 to 800 entries
        w = rng.integers(600, 801, n)
    elif kind == "some":
        w[:: 17] = rng.integers(200, 4000, w[::17].size)
    else:
        w[n // 2] = 9000
    m = n + 77
    rp = np.concatenate([[0], np.cumsum(w)]).astype(np.int32)
    ci = rng.integers(0, m, rp[-1]).astype(np.int32)
    v, x = rng.standard_normal(rp[-1]), rng.standard_normal(m)
    ref = np.zeros(n)
    for k in range(int(w.max())):
        on = w > k
        e = rp[:-1][on] + k
        ref[on] = ref[on] + v[e] * x[ci[e]]
    assert np.array_equal(sg.CSRMatrix(n, m, rp, ci, v).spmv(x), ref)


def test_few_long_rows_are_added_side_by_side(sg):
    """A block of 256 rows of 8,000 entries takes what one of 32 rows takes,
    times at most two: its eight warps add side by side, and the FP64 pipe, which
    serves them in turn (16 cycles each), is twice as long as one addition's
    latency (~80).  All rows one after another take eight times that."""
    import torch

    k = 8000
    rng = np.random.default_rng(1)
    runs = []
    for n in (32, 256):
        A = sg.CSRMatrix(n, n + 1, (k * np.arange(n + 1)).astype(np.int32),
                         rng.integers(0, n + 1, n * k).astype(np.int32), rng.standard_normal(n * k))
        x = torch.ones(n + 1, dtype=torch.float64, device="cuda")
        y = torch.empty(n, dtype=torch.float64, device="cuda")
        A.spmv(x, y)
        runs.append((A, x, y, []))
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(5):
        for A, x, y, ms in runs:
            torch.cuda.synchronize()
            a.record()
            A.spmv(x, y)  # returns with the product done
            b.record()
            b.synchronize()
            ms.append(a.elapsed_time(b))
    assert min(runs[1][3]) < 4 * min(runs[0][3])
