"""The work that a user of this package has it do, as cases that can be timed.

The package solves A x = b with preconditioned, restarted GMRES and FGMRES.
A program that uses it sets a preconditioner up, solves (one system or a
batch), applies the operator or the preconditioner by itself inside an outer
iteration of its own, sets up again for new coefficients, and trains and
applies the learned stage.  Matrices, partitions, vectors and weights are made
here with torch, so that `exact` knows them without the package.

Vectors are device tensors on one stream that torch and the package's context
share, unless a case says that it hands over host arrays.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import schwarz_gmres_dashboard_gb300 as sg

_stream = None


def _use_one_stream():
    """torch and the package's context work on one stream, as a program does
    that mixes the two without synchronising between them."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
        torch.cuda.set_stream(_stream)
        sg.default_context().set_stream(_stream.cuda_stream)


# ------------------------------------------------------------------ the cases
def _solve(nx, ny, nz=1, op="poisson", pc="ras", parts=(2, 2, 1), overlap=1, solver="gmres",
           restart=30, precision="fp64", factors="fp64", tol=1e-10, rule="abs", host=False):
    px, py, pz = parts
    return dict(kind="solve", nx=nx, ny=ny, nz=nz, op=op, pc=pc, px=px, py=py, pz=pz,
                overlap=overlap, solver=solver, restart=restart, precision=precision,
                factors=factors, tol=tol, rule=rule, host=host, field=1)


def listed():
    return [
        # the first program of a new user: a 400-row system in host arrays,
        # four subdomains
        dict(_solve(20, 20, host=True), name="poisson_20x20_ras4"),
        # the sizes of the published tables: a five-point grid with a handful
        # of subdomains, one ILU(0) block, and two-level FGMRES on a grid that
        # divides evenly into nothing
        dict(_solve(100, 100), name="poisson_100x100_ras4"),
        dict(_solve(128, 128, pc="ilu0", parts=(1, 1, 1)), name="poisson_128x128_ilu0"),
        dict(_solve(201, 187, pc="twolevel_ras", parts=(8, 4, 1), solver="fgmres"),
             name="poisson_201x187_fgmres_twolevel32"),
        # a 3D solve in FP64 throughout, wide overlap
        dict(_solve(64, 64, 64, parts=(4, 4, 4), overlap=2), name="poisson_64cubed_ras64"),
        # production: two million rows, variable coefficients, FP32 basis with
        # BF16 factors inside FP64 refinement, uneven subdomains
        dict(_solve(128, 128, 128, op="varcoef", pc="twolevel_ras", parts=(8, 8, 4),
                    precision="fp32", factors="bf16", tol=1e-12, rule="true"),
             name="varcoef_128cubed_mixed"),
        # many small anisotropic systems of uneven sizes, four right-hand sides
        dict(kind="batched", name="aniso_64_systems_x4", nsys=64, nmin=32, nmax=256, nrhs=4,
             precision="fp32", tol=1e-13, field=3),
        # the operator alone, on a ragged grid
        dict(kind="spmv", name="spmv_121x133x127", nx=121, ny=133, nz=127, op="varcoef", field=2),
        # the preconditioner alone, as an outer method of the user's own calls it
        dict(kind="apply", name="apply_128cubed_twolevel_bf16", nx=128, ny=128, nz=128,
             op="varcoef", pc="twolevel_ras", px=8, py=8, pz=4, overlap=1, factors="bf16", field=1),
        # a new coefficient field on a known pattern: upload, set-up, first apply
        dict(kind="resetup", name="resetup_64cubed_twolevel64", nx=64, ny=64, nz=64, op="varcoef",
             pc="twolevel_ras", px=4, py=4, pz=4, overlap=1, factors="fp32", field=1),
        # the learned stage: inside an apply, and one gradient of a training loop
        dict(kind="learned_apply", name="learned_apply_96cubed", nx=96, px=6, py=6, pz=3,
             factors="bf16", field=4),
        dict(kind="learned_gradient", name="learned_gradient_64cubed_x8", nx=64, batch=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve2d", "solve2d", "solve3d", "solve3d", "batched", "spmv", "apply",
                       "apply", "resetup", "learned_apply", "learned_gradient"])
    if kind == "solve2d":
        nx, ny = _log(rng, 16, 220), _log(rng, 16, 220)
        pc = rng.choice(["ras", "ras", "twolevel_ras", "ilu0"])
        if nx * ny > 17000 and pc == "ilu0":
            pc = "ras"
        parts = (rng.randint(1, max(1, min(8, nx // 8))), rng.randint(2, max(2, min(4, ny // 8))), 1)
        if pc == "ilu0":
            parts = (1, 1, 1)
        return _solve(nx, ny, op=rng.choice(["poisson", "aniso"]), pc=pc, parts=parts,
                      overlap=rng.randint(1, 2), solver=rng.choice(["gmres", "gmres", "fgmres"]),
                      restart=rng.choice([20, 30, 30, 40]), host=rng.random() < 0.25)
    if kind == "solve3d":
        mixed = rng.random() < 0.5
        hi = 120 if mixed else 72
        n = [_log(rng, 20, hi) for _ in range(3)]
        parts = tuple(max(1, min(8, round(v / rng.choice([12, 16, 20])))) for v in n)
        return _solve(*n, op=rng.choice(["poisson", "varcoef"]),
                      pc=rng.choice(["ras", "twolevel_ras"]), parts=parts,
                      overlap=rng.randint(1, 2) if max(n) < 80 else 1,
                      solver=rng.choice(["gmres", "gmres", "fgmres"]),
                      restart=rng.choice([20, 30, 30, 40]),
                      precision="fp32" if mixed else "fp64",
                      factors=rng.choice(["fp32", "bf16"]) if mixed else "fp64",
                      tol=1e-12 if mixed else 1e-10, rule="true" if mixed else "abs")
    if kind == "batched":
        return dict(kind="batched", nsys=_log(rng, 4, 60), nmin=32, nmax=rng.randint(64, 250),
                    nrhs=rng.choice([1, 2, 4, 4, 5]), precision=rng.choice(["fp32", "fp32", "fp64"]),
                    tol=1e-13, field=rng.randint(1, 9))
    if kind == "spmv":
        return dict(kind="spmv", nx=_log(rng, 16, 128), ny=_log(rng, 16, 128),
                    nz=_log(rng, 8, 128), op=rng.choice(["poisson", "varcoef", "graph"]),
                    field=rng.randint(1, 9))
    if kind in ("apply", "resetup"):
        f = rng.choice(["fp64", "fp32", "bf16"])
        d = dict(kind=kind, op="varcoef", pc=rng.choice(["ras", "twolevel_ras"]),
                 overlap=rng.randint(1, 2), factors=f, field=rng.randint(1, 9))
        if rng.random() < 0.3:
            nx, ny = _log(rng, 32, 250), _log(rng, 32, 250)
            return dict(d, op="aniso", nx=nx, ny=ny, nz=1, px=max(1, nx // 40),
                        py=max(1, ny // 40), pz=1)
        n = [_log(rng, 20, 96 if kind == "apply" else 64) for _ in range(3)]
        p = [max(1, min(8, round(v / 14))) for v in n]
        return dict(d, nx=n[0], ny=n[1], nz=n[2], px=p[0], py=p[1], pz=p[2])
    nx = 16 * rng.randint(2, 6)
    if kind == "learned_apply":
        return dict(kind=kind, nx=nx, px=rng.randint(2, 6), py=rng.randint(2, 6),
                    pz=rng.randint(2, 5), factors=rng.choice(["fp32", "bf16"]),
                    field=rng.randint(1, 9))
    return dict(kind=kind, nx=min(nx, 80), batch=rng.randint(1, 8 if nx <= 64 else 4))


# ------------------------------------------------------------------ matrices
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _uniform(shape, seed):
    return torch.rand(shape, generator=_gen(seed), dtype=torch.float64, device=_dev()) * 2 - 1


def _csr_of(cols, vals, on):
    """CSR from [n, w] columns in ascending order, values and a mask."""
    rp = torch.zeros(on.shape[0] + 1, dtype=torch.int64, device=on.device)
    rp[1:] = on.sum(1).cumsum(0)
    return rp, cols[on], vals[on]


def _grid_index(nx, ny, nz):
    z, y, x = torch.meshgrid(*(torch.arange(m, device=_dev()) for m in (nz, ny, nx)), indexing="ij")
    return x.reshape(-1), y.reshape(-1), z.reshape(-1)


def _stencil(nx, ny, nz, entries):
    """entries: (dx, dy, dz, value per row), sorted by their column."""
    x, y, z = _grid_index(nx, ny, nz)
    row = torch.arange(nx * ny * nz, device=_dev())
    cols, vals, on = [], [], []
    for dx, dy, dz, v in entries:
        ok = ((x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0)
              & (z + dz < nz))
        cols.append(row + (dz * ny + dy) * nx + dx)
        vals.append(torch.as_tensor(v, dtype=torch.float64, device=_dev()).expand(row.shape))
        on.append(ok)
    return _csr_of(torch.stack(cols, 1), torch.stack(vals, 1), torch.stack(on, 1))


def _poisson(nx, ny, nz):
    near = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    if nz == 1:
        near = [d for d in near if d[2] == 0]
    return _stencil(nx, ny, nz, [(*d, float(len(near) - 1) if d == (0, 0, 0) else -1.0) for d in near])


def _varcoef(nx, ny, nz, seed):
    """-div(k grad u), seven points, k the exponential of a smooth unit-variance
    random field, harmonic means on the faces, Dirichlet boundary."""
    w = torch.randn((nz, ny, nx), generator=_gen(seed), dtype=torch.float64, device=_dev())
    f = torch.fft.fftn(w)
    for d, m in enumerate((nz, ny, nx)):
        k = torch.fft.fftfreq(m, device=_dev(), dtype=torch.float64) * 2 * math.pi
        f = f * torch.exp(-(k * 4.0) ** 2 / 2).reshape([-1 if e == d else 1 for e in range(3)])
    g = torch.fft.ifftn(f).real
    k = torch.exp((g - g.mean()) / g.std())
    face = {}
    for d, name in ((2, "x"), (1, "y"), (0, "z")):
        lo = torch.roll(k, 1, d)
        face[name] = 2 * k * lo / (k + lo)

    def side(name, d, up):
        m = k.shape[d]
        v = torch.roll(face[name], -1, d) if up else face[name].clone()
        v.select(d, m - 1 if up else 0).copy_(k.select(d, m - 1 if up else 0))
        return v.reshape(-1)

    xl, xu, yl, yu, zl, zu = (side(a, d, u) for a, d in (("x", 2), ("y", 1), ("z", 0))
                              for u in (False, True))
    return _stencil(nx, ny, nz, [(0, 0, -1, -zl), (0, -1, 0, -yl), (-1, 0, 0, -xl),
                                 (0, 0, 0, xl + xu + yl + yu + zl + zu), (1, 0, 0, -xu),
                                 (0, 1, 0, -yu), (0, 0, 1, -zu)])


def _aniso(nx, ny, t, e):
    """-div(K grad u), nine points, K = diag(1, e) rotated by t."""
    c, s = math.cos(t), math.sin(t)
    a, b, m = c * c + e * s * s, s * s + e * c * c, (1 - e) * c * s
    return _stencil(nx, ny, 1, [(-1, -1, 0, -m / 2), (0, -1, 0, -b), (1, -1, 0, m / 2), (-1, 0, 0, -a),
                                (0, 0, 0, 2 * a + 2 * b), (1, 0, 0, -a), (-1, 1, 0, m / 2),
                                (0, 1, 0, -b), (1, 1, 0, -m / 2)])


def _graph(n, seed):
    """A weighted graph Laplacian plus the identity: uneven rows of 2 to 30
    neighbours, most of them near."""
    g = _gen(seed)
    deg = (2 + 28 * torch.rand(n, generator=g, device=_dev()) ** 4).long()
    row = torch.repeat_interleave(torch.arange(n, device=_dev()), deg)
    hop = torch.randn(row.shape, generator=g, device=_dev()).mul(300).long()
    col = (row + hop) % n
    key = torch.unique(torch.cat([row * n + col, col * n + row, torch.arange(n, device=_dev()) * (n + 1)]))
    r, c = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device=_dev())
    rp[1:] = torch.bincount(r, minlength=n).cumsum(0)
    d = (rp[1:] - rp[:-1]).double()
    v = torch.where(r == c, d[r], -1.0)
    return rp, c, v


def _matrix(case, seed=None):
    op, f = case.get("op", "varcoef"), case.get("field", 1) if seed is None else seed
    nx, ny, nz = case["nx"], case.get("ny", case["nx"]), case.get("nz", case["nx"])
    if op == "poisson":
        return _poisson(nx, ny, nz)
    if op == "aniso":
        return _aniso(nx, ny, 0.3 + 0.2 * (f % 5), 0.25)
    if op == "graph":
        return _graph(nx * ny * nz, f)
    return _varcoef(nx, ny, nz, f)


def _batch_sizes(case):
    r = np.random.RandomState(case["field"])
    return r.randint(case["nmin"], case["nmax"] + 1, case["nsys"]), r


def _batch(case):
    """Block-diagonal union of square anisotropic systems of uneven sizes,
    their row offsets, and a partition of 4 to 16 boxes in each."""
    sizes, r = _batch_sizes(case)
    rps, cis, vs, parts, rows, nnz, np_ = [], [], [], [], [0], 0, 0
    for k in sizes:
        rp, ci, v = _aniso(int(k), int(k), r.uniform(0, math.pi), 10 ** r.uniform(-3, 0))
        rps.append(rp[:-1] + nnz)
        cis.append(ci + rows[-1])
        vs.append(v)
        rows.append(rows[-1] + int(k) ** 2)
        nnz += len(ci)
        side = 2 if k < 150 else 3 if k < 220 else 4
        part, p = _partition(dict(nx=int(k), ny=int(k), nz=1, px=side, py=side, pz=1))
        parts.append(part + np_)
        np_ += p
    rps.append(torch.tensor([nnz], device=_dev()))
    return ((torch.cat(rps), torch.cat(cis), torch.cat(vs)), np.array(rows, np.int32),
            np.concatenate(parts).astype(np.int32), np_)


def _cuts(n, p, seed):
    """p uneven pieces of n cells: the piece of every cell."""
    r = np.random.RandomState(seed)
    p = max(1, min(p, n // 2))
    at = np.round(np.arange(1, p) * n / p + r.uniform(-0.15, 0.15, p - 1) * n / p).astype(int)
    piece = np.zeros(n, np.int64)
    for a in at:
        piece[a:] += 1
    return piece, p


def _partition(case):
    nx, ny, nz = case["nx"], case.get("ny", case["nx"]), case.get("nz", case["nx"])
    ax, px = _cuts(nx, case["px"], 11)
    ay, py = _cuts(ny, case["py"], 12)
    az, pz = _cuts(nz, case["pz"], 13)
    part = (az[:, None, None] * py + ay[None, :, None]) * px + ax[None, None, :]
    return part.reshape(-1).astype(np.int32), px * py * pz


def _csr(m):
    rp, ci, v = m
    return sg.CSRMatrix(len(rp) - 1, len(rp) - 1, rp.int().cpu().numpy(), ci.int().cpu().numpy(),
                        v.cpu().numpy())


def _precond(case):
    t = {"fp64": (sg.FP64, sg.FP64), "fp32": (sg.FP32, sg.FP32), "bf16": (sg.BF16, sg.FP32)}
    fd, sd = t[case["factors"]]
    if case.get("pc") == "ilu0":
        return sg.ILU0Precond(fd, sd)
    part, np_ = _partition(case)
    if case.get("pc", "twolevel_ras") == "ras":
        return sg.RASPrecond(np_, case.get("overlap", 1), part, fd, sd)
    return sg.TwoLevelSchwarzPrecond(np_, case.get("overlap", 1), sg.FineLevelType.RAS, part, fd, sd)


# ------------------------------------------------------------------ one pass
NET = 4 * (27 * 256 + 16)  # parameters of the learned stage's network


def _weights(seed):
    """Four 3x3x3 layers in the layout [27][in][out], 16 biases after each;
    channels that the first and the last layer do not have stay zero."""
    r = np.random.RandomState(seed)
    w = np.zeros(NET + 1, np.float32)
    for k, (ci, co) in enumerate([(2, 16), (16, 16), (16, 16), (16, 1)]):
        at = k * (27 * 256 + 16)
        m = np.zeros((27, 16, 16), np.float32)
        m[:, :ci, :co] = r.randn(27, ci, co) * math.sqrt(2.0 / (27 * ci))
        b = np.zeros(16, np.float32)
        b[:co] = 0.05 * r.randn(co)
        w[at: at + 27 * 256] = m.reshape(-1)
        w[at + 27 * 256: at + 27 * 256 + 16] = b
    w[NET] = 0.1
    return w


def _samples(case, seed):
    r = np.random.RandomState(seed)
    nc = (case["nx"] // 2) ** 3
    return (r.randn(case["batch"], nc, 2).astype(np.float32),
            r.randn(case["batch"], nc).astype(np.float32))


def prepare(case, seed):
    _use_one_stream()
    kind = case["kind"]
    if kind == "learned_gradient":
        stage = sg.LearnedCorrection(case["nx"])
        stage.weights = _weights(5)
        x, t = _samples(case, seed)
        return dict(kind=kind, stage=stage, x=x, t=t)
    if kind == "batched":
        m, rows, part, nparts = _batch(case)
        A = _csr(m).upload()
        dt = sg.FP32 if case["precision"] == "fp32" else sg.FP64
        M = sg.RASPrecond(nparts, 1, part, dt, dt)
        M.setup(A)
        X = _uniform((case["nrhs"], A.nrows), seed)  # the solutions
        B = torch.empty_like(X)
        for k in range(case["nrhs"]):
            A.spmv(X[k], B[k])
        p = sg.GMRESParams(restart=30, max_iter=2000, tol=case["tol"], tol_kind=sg.TOL_TRUE_REL,
                           precision=dt)
        return dict(kind=kind, A=A, M=M, sys=rows, nrhs=case["nrhs"], B=B, p=p)
    A = _csr(_matrix(case)).upload()
    v = _uniform(A.nrows, seed)
    if kind == "spmv":
        return dict(kind=kind, A=A, x=v, y=torch.empty_like(v))
    M = _precond(case)
    M.setup(A)
    st = dict(kind=kind, A=A, M=M, x=v, y=torch.empty_like(v))
    if kind == "resetup":
        st["vals"] = _matrix(case, 1000 + seed)[2].cpu().numpy()
    elif kind == "learned_apply":
        stage = sg.LearnedCorrection(case["nx"])
        stage.set_matrix(A)
        stage.weights = _weights(5)
        stage.attach(M)
        st["stage"] = stage
    elif kind == "solve":
        b = torch.empty_like(v)
        A.spmv(v, b)  # the solution is v
        st.update(b=b.cpu().numpy() if case["host"] else b, host=case["host"],
                  solver=sg.fgmres if case["solver"] == "fgmres" else sg.gmres,
                  p=sg.GMRESParams(restart=case["restart"], max_iter=3000, tol=case["tol"],
                                   tol_kind=sg.TOL_TRUE_REL if case["rule"] == "true"
                                   else sg.TOL_REF_ABS,
                                   precision=sg.FP32 if case["precision"] == "fp32" else sg.FP64))
    return st


def run(st):
    kind = st["kind"]
    if kind == "solve":
        x = np.zeros(st["A"].nrows) if st["host"] else torch.zeros_like(st["b"])
        st["solver"](st["A"], st["b"], x, st["M"], st["p"])
        return x
    if kind == "batched":
        X = torch.zeros_like(st["B"])
        sg.solve_batched(st["A"], st["M"], st["sys"], st["nrhs"], st["B"], X, st["p"])
        return X
    if kind == "spmv":
        return st["A"].spmv(st["x"], st["y"])
    if kind == "learned_gradient":
        loss, g = st["stage"].gradient(st["x"], st["t"])
        return {"loss": loss, "gradient": g}
    if kind == "resetup":
        st["A"].vals = st["vals"]
        st["A"].upload()
        st["M"].setup(st["A"])
    return st["M"].apply(st["x"], st["y"])


# ------------------------------------------------------------------ its work
def work(case):
    """Inputs once, outputs once; for a solve the operations of a typical
    number of iterations."""
    kind = case["kind"]
    if kind == "learned_gradient":
        v = (case["nx"] // 2) ** 3 * case["batch"]
        return {"bytes": v * 12 + NET * 8, "flops": 3 * 2 * v * 27 * (2 * 16 + 256 + 256 + 16)}
    if kind == "batched":
        n = case["nsys"] * (case["nmin"] + case["nmax"]) ** 2 / 4
        return {"bytes": n * (9 * 12 + 9 * 8) + n * case["nrhs"] * 16,
                "flops": n * case["nrhs"] * 150 * (4 * 9 + 8 * 15)}
    n = case["nx"] * case.get("ny", case["nx"]) * case.get("nz", case["nx"])
    w = {"poisson": 5 if case.get("nz", 0) == 1 else 7, "aniso": 9, "graph": 14}.get(case.get("op"), 7)
    vb = {"fp64": 8, "fp32": 4, "bf16": 2}.get(case.get("factors"), 8)
    if kind == "spmv":
        return {"bytes": n * (w * 12 + 20), "flops": 2 * w * n}
    apply = {"bytes": n * (w * (vb + 4) + 20), "flops": 2 * w * n}
    if kind == "apply":
        return apply
    if kind == "resetup":
        return {"bytes": 2 * n * w * 12 + apply["bytes"], "flops": n * w * w + apply["flops"]}
    if kind == "learned_apply":
        v = n // 8
        return {"bytes": apply["bytes"] + n * (w * 8 + 16), "flops": 2 * v * 27 * (2 * 16 + 256 + 256 + 16)
                + 2 * apply["flops"]}
    m = case["restart"]
    return {"bytes": n * (w * 12 + 20) + apply["bytes"], "flops": 100 * n * (4 * w + 4 * m)}


# ------------------------------------------------------------------ 64-bit values
def _spmv64(m, x):
    rp, ci, v = m
    row = torch.repeat_interleave(torch.arange(len(rp) - 1, device=v.device), rp[1:] - rp[:-1])
    return torch.zeros_like(x).index_add_(0, row, v * x[ci])


def _levels(cols, on):
    """Level of every row: one above the highest row that it depends on."""
    lev = torch.zeros(cols.shape[0], dtype=torch.int64, device=cols.device)
    while True:
        new = torch.where(on, lev[cols] + 1, 0).amax(1)
        if torch.equal(new, lev):
            return [torch.nonzero(lev == k)[:, 0] for k in range(int(lev.max()) + 1)]
        lev = new


def _schwarz64(m, part, nparts, overlap, x, coarse):
    """Restricted additive Schwarz with ILU(0) blocks, and the piecewise
    constant coarse term, all subdomains side by side."""
    rp, ci, v = m
    n, dev = len(rp) - 1, v.device
    part = torch.as_tensor(part.astype(np.int64), device=dev)
    deg = rp[1:] - rp[:-1]
    row = torch.repeat_interleave(torch.arange(n, device=dev), deg)
    w = int(deg.max())
    pos = torch.arange(len(ci), device=dev) - rp[row]
    gc = torch.full((n, w), -1, dtype=torch.int64, device=dev)
    gv = torch.zeros((n, w), dtype=torch.float64, device=dev)
    gc[row, pos], gv[row, pos] = ci, v
    key = part * n + torch.arange(n, device=dev)
    for _ in range(overlap):  # the neighbours of every member join
        r, p = key % n, key // n
        near = gc[r]
        key = torch.unique(torch.cat([key, (p[:, None] * n + near)[near >= 0]]))
    key = torch.unique(key)
    r, p = key % n, key // n
    N = len(key)
    want = p[:, None] * n + gc[r]
    at = torch.searchsorted(key, want).clamp(max=N - 1)
    has = (gc[r] >= 0) & (key[at] == want)
    me = torch.arange(N, device=dev)[:, None]
    col, val = torch.where(has, at, -1), torch.where(has, gv[r], 0.0)
    low, up = has & (col < me), has & (col > me)
    dpos = (col == me).long().argmax(1)
    safe = col.clamp(min=0)
    flev = _levels(safe, low)
    for R in flev:
        for j in range(w):
            k = safe[R, j]
            a = torch.where(low[R, j], val[R, j] / val[k, dpos[k]], val[R, j])
            val[R, j] = a
            for q in range(w):
                hit = (col[R] == col[k, q][:, None]) & (low[R, j] & up[k, q])[:, None]
                val[R] = val[R] - torch.where(hit, (a * val[k, q])[:, None], 0.0)
    t = x[r].clone()
    for R in flev:
        t[R] = t[R] - (torch.where(low[R], val[R], 0.0) * t[safe[R]]).sum(1)
    for R in _levels(safe, up):
        t[R] = (t[R] - (torch.where(up[R], val[R], 0.0) * t[safe[R]]).sum(1)) / val[R, dpos[R]]
    own = part[r] == p
    y = torch.zeros_like(x)
    y[r[own]] = t[own]
    if coarse:
        c = 1.0 / torch.bincount(part, minlength=nparts).double().sqrt()
        a0 = torch.zeros(nparts * nparts, dtype=torch.float64, device=dev)
        a0.index_add_(0, part[row] * nparts + part[ci], c[part[row]] * v * c[part[ci]])
        r0 = torch.zeros(nparts, dtype=torch.float64, device=dev).index_add_(0, part, c[part] * x)
        y = y + (c * torch.linalg.solve(a0.reshape(nparts, nparts), r0))[part]
    return y


def _net64(w, x):
    """The learned stage's network on [batch, 2, D, D, D]."""
    for k in range(4):
        at = k * (27 * 256 + 16)
        m = w[at: at + 27 * 256].reshape(3, 3, 3, 16, 16).permute(4, 3, 0, 1, 2)
        if k == 0:
            m = m[:, :2]
        b = w[at + 27 * 256: at + 27 * 256 + 16]
        x = torch.nn.functional.conv3d(x, m, b, padding=1)
        if k < 3:
            x = torch.relu(x)
    return x[:, :1]


def _up64(y):
    """Cell-centred trilinear prolongation of [D, D, D]."""
    for d in range(3):
        m = y.shape[d]
        at = torch.arange(m, device=y.device)
        near = 0.75 * y
        lo = near + 0.25 * y.index_select(d, (at - 1).clamp(min=0))
        hi = near + 0.25 * y.index_select(d, (at + 1).clamp(max=m - 1))
        y = torch.stack([lo, hi], d + 1).flatten(d, d + 1)
    return y


def _down64(v, nx):
    return v.reshape(nx // 2, 2, nx // 2, 2, nx // 2, 2).mean((1, 3, 5))


def exact(case, seed):
    kind = case["kind"]
    torch.backends.cudnn.allow_tf32 = False
    if kind == "learned_gradient":
        D = case["nx"] // 2
        x, t = (torch.as_tensor(a, device=_dev()).double() for a in _samples(case, seed))
        w = torch.as_tensor(_weights(5)[:NET], device=_dev()).double().requires_grad_()
        y = _net64(w, x.reshape(-1, D, D, D, 2).permute(0, 4, 1, 2, 3)).reshape(t.shape)
        loss = ((y - t) ** 2).mean()
        loss.backward()
        g = w.grad.clone()
        for k in (0, 3):  # the channels that these layers do not have
            at = k * (27 * 256 + 16)
            m = g[at: at + 27 * 256].reshape(27, 16, 16)
            if k == 0:
                m[:, 2:] = 0
            else:
                m[:, :, 1:] = 0
                g[at + 27 * 256 + 1: at + 27 * 256 + 16] = 0
        return {"loss": float(loss), "gradient": g}
    if kind == "batched":
        return _uniform((case["nrhs"], int((_batch_sizes(case)[0] ** 2).sum())), seed)
    n = case["nx"] * case.get("ny", case["nx"]) * case.get("nz", case["nx"])
    x = _uniform(n, seed)
    if kind == "solve":
        return x.cpu().numpy() if case["host"] else x
    m = _matrix(case, 1000 + seed if kind == "resetup" else None)
    if kind == "spmv":
        return _spmv64(m, x)
    part, nparts = _partition(case)
    coarse = case.get("pc", "twolevel_ras") == "twolevel_ras"
    z = _schwarz64(m, part, nparts, case.get("overlap", 1), x, coarse)
    if kind == "learned_apply":
        nx = case["nx"]
        rc = _down64(x - _spmv64(m, z), nx)
        s = rc.square().mean().sqrt()
        rp, ci, v = m
        row = torch.repeat_interleave(torch.arange(n, device=v.device), rp[1:] - rp[:-1])
        f = _down64(torch.log(v[row == ci]), nx)
        f = (f - f.mean()) / f.std(correction=0)
        w = torch.as_tensor(_weights(5), device=_dev()).double()
        y = _net64(w[:NET], torch.stack([rc / s, f])[None])[0, 0]
        z = z + s * w[NET] * _up64(y).reshape(-1)
    return z
