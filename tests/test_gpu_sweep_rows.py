"""The level records of the TMA-fed sweep: row structs (2, 3 and 4 nonzeros per
triangle) and component records (other widths, or a subdomain so near the
shared-memory limit that only the smaller records fit), levels of fewer, as
many and more rows than the level threads.  FP64 applies equal the oracle bit
for bit; FP32 and BF16 factors equal the barrier-per-level sweep bit for bit
(both round every multiply-add once and multiply by the FP32 reciprocal)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(sg, n, extra, seed):
    """Symmetric pattern, diagonally dominant, `extra` random couplings a row."""
    r = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), extra)
    j = (i + r.integers(1, 40, i.size)) % n
    key = np.unique(np.concatenate([i * n + j, j * n + i, np.arange(n) * (n + 1)]))
    row, col = key // n, key % n
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    deg = np.diff(rp)
    v = np.where(row == col, deg[row].astype(float), -1.0 + 0.1 * r.random(row.size))
    return sg.CSRMatrix(n, n, rp, col.astype(np.int32), v)


def _case(sg, name):
    if name == "5pt":
        A, g = sg.make_poisson_2d(67, 45), (67, 45, 1)
    elif name == "7pt":
        A, g = sg.make_varcoef_3d(23, 20, 17, 1.0, 4.0, 3), (23, 20, 17)
    elif name == "9pt":
        A, g = sg.make_aniso_2d(50, 71, 0.3, 0.6), (50, 71, 1)
    elif name == "tridiagonal":
        return sg.make_poisson_2d(300, 1), np.repeat(np.arange(3), 100).astype(np.int32), 3
    else:
        A = _graph(sg, 1500, 4, 7)
        return A, sg.partition_graph(A, 5), 5
    return A, sg.partition_boxes(*g, 5, 0.1, seed=2), 5


@pytest.mark.parametrize("name", ["5pt", "7pt", "9pt", "tridiagonal", "graph"])
@pytest.mark.parametrize("threads", [0, 32, 64, 128, 512])
@pytest.mark.parametrize("dt", ["fp64", "fp32", "bf16"])
def test_rows_and_passes(sg, oracle, name, threads, dt):
    A, part, p = _case(sg, name)
    fd, sd = {"fp64": (sg.FP64, sg.FP64), "fp32": (sg.FP32, sg.FP32),
              "bf16": (sg.BF16, sg.FP32)}[dt]
    x = sg.uniform(A.nrows, 11)
    pc = sg.RASPrecond(p, 1, part, fd, sd, sweep_threads=threads)
    pc.setup(A)
    assert pc.sweep_choice()["sweep"] == "tma" and pc.check() == 0
    y = pc.apply(x)
    if dt == "fp64":
        assert np.array_equal(y, oracle.precond("ras", A, p, 1, part).apply(x))
    else:
        ref = sg.RASPrecond(p, 1, part, fd, sd, sweep="level")
        ref.setup(A)
        assert np.array_equal(y, ref.apply(x))


@pytest.mark.parametrize("edge", [128, 150, 159, 162, 164])
def test_one_block_near_the_shared_memory_limit(sg, oracle, edge):
    A = sg.make_poisson_2d(edge, edge)
    x = sg.uniform(A.nrows, 12)
    pc = sg.ILU0Precond()
    pc.setup(A)
    assert pc.check() == 0
    assert np.array_equal(pc.apply(x), oracle.precond("ilu0", A).apply(x))
    # the solver's sweeps multiply by the rounded reciprocal: one rounding
    # (2^-53) more per row than the division, so a solve to 1e-10 must agree
    b = A.spmv(x)
    s = np.zeros(A.nrows)
    r = sg.gmres(A, b, s, pc, sg.GMRESParams(restart=30, max_iter=2000, tol=1e-12,
                                             tol_kind=sg.TOL_TRUE_REL))
    assert r.converged and r.true_rel_residual <= 1e-12
