"""FGMRES whose preconditioner gives directions that repeat or span few
dimensions: no step can reduce the residual once they are used up, and none may
raise it.  The two-pass orthogonalisation ends a cycle at a vector that lies in
the span of those before; ones that it has no reason to end converge as with
three passes."""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as sl

pytestmark = pytest.mark.gpu

N = 30


def _preconditioners(S, n):
    rng = np.random.default_rng(0)
    U, F = rng.standard_normal((n, 3)), rng.standard_normal((5, n))
    Q = np.kron(np.eye(9), np.ones((n // 9, 1))) / np.sqrt(n // 9)
    E = np.linalg.inv(Q.T @ (S @ Q))
    calls = [0]

    def turns(k):
        def f(r):
            calls[0] += 1
            return U[:, calls[0] % k]
        return f

    return {"one": lambda r: np.ones_like(r), "two": turns(2), "three": turns(3),
            "rank1": lambda r: U[:, 0] * (F[0] @ r), "rank5": lambda r: F.T @ (F @ r) / n,
            "coarse": lambda r: Q @ (E @ (Q.T @ r))}


def _solve(sg, A, f, b, precision, ortho=0):
    H = sg.HostPreconditioner(lambda u, w: w.__setitem__(slice(None), f(u)), A.nrows)
    x = np.zeros(A.nrows)
    r = sg.fgmres(A, b, x, H, sg.GMRESParams(restart=20, max_iter=60, tol=1e-10, ortho=ortho,
                                             tol_kind=sg.TOL_TRUE_REL, precision=precision))
    return x, r


@pytest.mark.parametrize("name", ["one", "two", "three", "rank1", "rank5", "coarse"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_dependent_directions(sg, name, precision):
    A = sg.make_poisson_2d(N, N)
    S = sp.csr_matrix((A.vals, A.col_idx, A.row_ptr), shape=(A.nrows, A.nrows))
    b = sg.uniform(A.nrows, 3)
    x, r = _solve(sg, A, _preconditioners(S, A.nrows)[name], b,
                  sg.FP64 if precision == "fp64" else sg.FP32)
    # from 1: a column of noise adds its coefficient times the rounding of its
    # direction, the residual's size, in each of three cycles
    assert np.linalg.norm(b - S @ x) <= 4 * np.linalg.norm(b)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind", ["exact", "nearly", "half"])
def test_strong_preconditioners_converge_alike(sg, kind, precision):
    A = sg.make_poisson_2d(N, N)
    S = sp.csr_matrix((A.vals, A.col_idx, A.row_ptr), shape=(A.nrows, A.nrows))
    b = sg.uniform(A.nrows, 3)
    lu = sl.splu(S.tocsc())
    f = {"exact": lu.solve, "nearly": lambda r: lu.solve(r) * (1 + 1e-6 * np.sign(r)),
         "half": lambda r: lu.solve(r).astype(np.float16).astype(float)}[kind]
    p = sg.FP64 if precision == "fp64" else sg.FP32
    x, r = _solve(sg, A, f, b, p)
    y, q = _solve(sg, A, f, b, p, ortho=1)
    assert r.converged and q.converged and abs(r.iterations - q.iterations) <= 1
    # unreachable tolerance: the solution is kept once it is there
    H = sg.HostPreconditioner(lambda u, w: w.__setitem__(slice(None), f(u)), A.nrows)
    z = np.zeros(A.nrows)
    sg.fgmres(A, b, z, H, sg.GMRESParams(restart=20, max_iter=40, tol=1e-300, precision=p))
    assert np.linalg.norm(b - S @ z) <= 1e-10 * np.linalg.norm(b)
