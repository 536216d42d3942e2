"""Threads with contexts of their own, whose preconditioners need different
amounts of shared memory: set-ups, applies and solves give what they give one
after another, bit for bit."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _work(sg, k, sweep, two_level, out):
    ctx = sg.Context(0)
    A = sg.make_poisson_2d(40 + k, 31)
    n = A.nrows
    part = (np.arange(n) * 6 // n).astype(np.int32)
    for it in range(8):
        dt = (sg.FP64, sg.FP32)[it % 2]
        if two_level:
            M = sg.TwoLevelSchwarzPrecond(6, 1, sg.FineLevelType.RAS, part, dt, dt, ctx=ctx, sweep=sweep)
        else:
            M = sg.RASPrecond(6, 1, part, dt, dt, ctx=ctx, sweep=sweep)
        A.upload(ctx)
        M.setup(A)
        b, x = sg.uniform(n, it), np.zeros(n)
        (sg.gmres, sg.fgmres)[it % 2](A, b, x, M, sg.GMRESParams(
            restart=(20, 33)[it % 2], max_iter=100, tol=1e-9, tol_kind=sg.TOL_TRUE_REL, precision=dt))
        out += [x, M.apply(b), A.spmv(b)]


@pytest.mark.parametrize("sweep", ["tma", "level", "syncfree"])
@pytest.mark.parametrize("two_level", [False, True])
def test_threads_do_not_disturb_each_other(sg, sweep, two_level):
    errors = []

    def run(k, out):
        try:
            _work(sg, k, sweep, two_level, out)
        except Exception as e:  # reported below, with the thread's number
            errors.append((k, str(e)))

    for _ in range(3):
        together = [[] for _ in range(5)]
        threads = [threading.Thread(target=run, args=(k, together[k])) for k in range(5)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        for k in range(5):
            alone = []
            _work(sg, k, sweep, two_level, alone)
            assert len(alone) == len(together[k])
            assert all(np.array_equal(a, b) for a, b in zip(alone, together[k]))
