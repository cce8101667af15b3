"""Performance cases of the sparse solve path, through the public Python API.

A case is a dict of plain values; ``prepare`` makes what a user's program
holds before the call (matrix, preconditioner, vectors, made from the seed),
``run`` is one pass, ``exact`` the same result in 64 bits with torch / numpy
alone.  Kinds:

  mult    y (=, +=) A x of a CSR, ELL or banded matrix
  apply   y = P^-1 x of an ILU(0) / IC(0) preconditioner
  solve   one Krylov solve from x = 0 with a preconditioner at hand
  step    preconditioner set-up and a mixed-precision solve (what a program
          pays whose matrix changes from solve to solve)
  batch   a batch of uneven systems, from host arrays to host solutions

Matrices: grid operators in natural order (2D 5-point, 3D 7-point; diffusion
with log-normal cell coefficients, optionally with convection), 2D 9-point
operators, and irregular matrices with power-law row lengths.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from mtl4_b200 import itl, mtl, serve

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
TORCH = {"f64": torch.float64, "f32": torch.float32}
NUMPY = {"f64": np.float64, "f32": np.float32}


def listed():
    return [
        # the smallest call: one product on a grid of about a thousand points (launch and call overhead)
        dict(name="mult_2d_33x31_f64", kind="mult", matrix="grid2d", nx=33, ny=31, nz=1, fmt="csr", dtype="f64",
             assign="="),
        # the stencil product of every 3D solve
        dict(name="mult_3d_128_f64", kind="mult", matrix="grid3d", nx=128, ny=128, nz=128, fmt="csr", dtype="f64",
             assign="="),
        # an irregular matrix (web- or network-like): 4M rows, about 40M entries at random columns
        dict(name="mult_powerlaw_4M_f64", kind="mult", matrix="powerlaw", nx=4194304, ny=1, nz=1, fmt="csr",
             dtype="f64", assign="="),
        # FP32 preconditioner apply inside mixed-precision solves, 3D convection-diffusion
        dict(name="ilu0_3d_128_f32", kind="apply", matrix="grid3d", nx=128, ny=128, nz=128, pc="ilu_0", dtype="f32",
             storage="f32"),
        # FP64 apply on a ragged 2D grid
        dict(name="ic0_2d_1001x777_f64", kind="apply", matrix="grid2d", nx=1001, ny=777, nz=1, pc="ic_0", dtype="f64",
             storage="f64"),
        # an operator that is no 5- or 7-point stencil
        dict(name="ilu0_9pt_317x255_f64", kind="apply", matrix="nine", nx=317, ny=255, nz=1, pc="ilu_0", dtype="f64",
             storage="f64"),
        # CG with the diagonal preconditioner on the 256 x 256 Laplacian: hundreds of short iterations
        dict(name="cg_diagonal_2d_256", kind="solve", matrix="laplace2d", nx=256, ny=256, nz=1, solver="cg",
             pc="diagonal", rtol=1e-8, beta=0.0),
        # CG with IC(0) on a 3D variable-coefficient operator of odd sides
        dict(name="cg_ic0_3d_65x50x41", kind="solve", matrix="grid3d", nx=65, ny=50, nz=41, solver="cg", pc="ic_0",
             rtol=1e-8, beta=0.0),
        # BiCGSTAB with ILU(0) in FP64 on 128^3 convection-diffusion
        dict(name="bicgstab_ilu0_3d_128", kind="solve", matrix="convdiff3d", nx=128, ny=128, nz=128,
             solver="bicgstab", pc="ilu_0", rtol=1e-8, beta=0.0),
        # restarted GMRES with ILU(0)
        dict(name="gmres_ilu0_3d_48", kind="solve", matrix="convdiff3d", nx=48, ny=48, nz=48, solver="gmres",
             pc="ilu_0", rtol=1e-8, beta=0.0),
        # set-up and mixed-precision BiCGSTAB on 128^3 convection-diffusion
        dict(name="step_ilu0_3d_128", kind="step", matrix="convdiff3d", nx=128, ny=128, nz=128, solver="bicgstab",
             pc="ilu_0", rtol=1e-8, beta=0.0),
        # uneven 2D and 3D systems with diagonal and IC(0) preconditioners solved together
        dict(name="batch_24_f64", kind="batch", count=24, lo=1000, hi=100000, mixed=False, rtol=1e-8, spread=4),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mult", "mult", "apply", "apply", "apply", "solve", "solve", "step", "batch"])
    if kind == "mult":
        m = rng.choice(["grid2d", "grid3d", "powerlaw", "nine"])
        fmt = "csr" if m == "powerlaw" else rng.choice(["csr", "csr", "ell", "banded"])
        nx, ny, nz = {"grid2d": lambda: (_logint(rng, 16, 1500), _logint(rng, 16, 1500), 1),
                      "grid3d": lambda: (_logint(rng, 8, 128), _logint(rng, 8, 128), _logint(rng, 8, 128)),
                      "powerlaw": lambda: (_logint(rng, 1000, 2000000), 1, 1),
                      "nine": lambda: (_logint(rng, 16, 1000), _logint(rng, 16, 1000), 1)}[m]()
        return dict(kind="mult", matrix=m, nx=nx, ny=ny, nz=nz, fmt=fmt, dtype=rng.choice(["f64", "f64", "f32"]),
                    assign=rng.choice(["=", "=", "+="]))
    if kind == "apply":
        m = rng.choice(["grid2d", "grid3d", "grid3d", "nine"])
        nx, ny, nz = {"grid2d": lambda: (_logint(rng, 24, 1200), _logint(rng, 24, 1200), 1),
                      "grid3d": lambda: (_logint(rng, 12, 128), _logint(rng, 12, 128), _logint(rng, 12, 128)),
                      "nine": lambda: (_logint(rng, 24, 400), _logint(rng, 24, 400), 1)}[m]()
        dt = rng.choice(["f64", "f32"])
        return dict(kind="apply", matrix=m, nx=nx, ny=ny, nz=nz, pc="ilu_0" if m == "nine" else rng.choice(["ilu_0", "ic_0"]),
                    dtype=dt, storage="f32" if dt == "f32" else rng.choice(["f64", "f64", "f32"]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 40), lo=_logint(rng, 500, 2000), hi=_logint(rng, 20000, 100000),
                    mixed=rng.random() < 0.5, rtol=1e-8, spread=rng.randint(0, 1000))
    three = rng.random() < 0.5
    nx, ny, nz = ((_logint(rng, 12, 90), _logint(rng, 12, 90), _logint(rng, 12, 90)) if three
                  else (_logint(rng, 24, 400), _logint(rng, 24, 400), 1))
    conv = kind == "step" or rng.random() < 0.5
    solver = rng.choice(["bicgstab", "bicgstab", "gmres"]) if kind == "solve" and conv else "bicgstab" if conv else "cg"
    pc = "ilu_0" if conv else rng.choice(["ic_0", "diagonal"])
    return dict(kind=kind, matrix="grid3d" if three else "grid2d", nx=nx, ny=ny, nz=nz, solver=solver, pc=pc,
                rtol=1e-8, beta=0.3 if conv else 0.0)


# ------------------------------------------------------------------ matrices
# A grid matrix is (stencil directions in ascending column order, one value
# array per direction on the grid [nz, ny, nx], zero where the neighbour is
# missing); its CSR holds the entries inside the grid.

def _directions(m):
    if m == "nine":
        return [(dx, dy, 0) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    if m in ("grid2d", "laplace2d"):
        return [(0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0)]
    return [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]


def _inside(d, shape):
    """Mask [nz, ny, nx] of the points whose neighbour in direction d exists."""
    m = torch.ones(shape, dtype=torch.bool, device=DEV)
    for axis, s in ((2, d[0]), (1, d[1]), (0, d[2])):
        if s < 0:
            m.narrow(axis, 0, min(-s, shape[axis])).fill_(False)
        elif s > 0:
            m.narrow(axis, max(shape[axis] - s, 0), min(s, shape[axis])).fill_(False)
    return m


def _shifted(a, d):
    """a at the neighbour in direction d (the point's own value outside the grid)."""
    out = a.clone()
    nz, ny, nx = a.shape
    x0, x1, y0, y1, z0, z1 = max(0, -d[0]), nx - max(0, d[0]), max(0, -d[1]), ny - max(0, d[1]), max(0, -d[2]), nz - max(0, d[2])
    if x1 > x0 and y1 > y0 and z1 > z0:
        out[z0:z1, y0:y1, x0:x1] = a[z0 + d[2]:z1 + d[2], y0 + d[1]:y1 + d[1], x0 + d[0]:x1 + d[0]]
    return out


def _grid_values(matrix, nx, ny, nz, g, beta):
    """Values per direction: diffusion between a cell and its neighbours
    (mean of the two coefficients; a boundary face takes the cell's own and
    adds to the diagonal only), plus centred convection of strength beta."""
    shape = (nz, ny, nx)
    dirs = _directions(matrix)
    if matrix == "convdiff3d":
        h = 1.0 / (nx + 1)
        wind, kappa, scale = (0.5, 0.3, 0.2), torch.ones(shape, dtype=torch.float64, device=DEV), 1.0 / (h * h)
    elif matrix == "laplace2d":
        h, wind, kappa, scale = 1.0, (0.0, 0.0, 0.0), torch.ones(shape, dtype=torch.float64, device=DEV), 1.0
    else:
        h, wind, scale = 1.0, (0.5 * beta, 0.3 * beta, 0.2 * beta), 1.0
        kappa = torch.exp(0.5 * torch.randn(shape, generator=g, dtype=torch.float64, device=DEV))
    vals, diag = {}, torch.zeros(shape, dtype=torch.float64, device=DEV)
    for d in dirs:
        if d == (0, 0, 0):
            continue
        weight = 1.0 if abs(d[0]) + abs(d[1]) + abs(d[2]) == 1 else 0.25
        face = weight * scale * 0.5 * (kappa + _shifted(kappa, d))
        diag += face
        conv = sum(s * w for s, w in zip(d, wind)) / (2 * h) if weight == 1.0 else 0.0
        vals[d] = torch.where(_inside(d, shape), -face + conv, torch.zeros((), dtype=torch.float64, device=DEV))
    vals[(0, 0, 0)] = diag
    return dirs, vals


def _grid_csr(matrix, nx, ny, nz, g, beta=0.0):
    shape, n = (nz, ny, nx), nx * ny * nz
    dirs, vals = _grid_values(matrix, nx, ny, nz, g, beta)
    mask = torch.stack([_inside(d, shape).reshape(-1) for d in dirs], 1)
    rows = torch.arange(n, device=DEV)
    cols = torch.stack([rows + d[0] + nx * (d[1] + ny * d[2]) for d in dirs], 1)[mask]
    data = torch.stack([vals[d].reshape(-1) for d in dirs], 1)[mask]
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(mask.sum(1), 0, out=rp[1:])
    return SimpleNamespace(n=n, rp=rp, col=cols.to(torch.int32), val=data, dirs=dirs, grid=vals)


def _powerlaw_csr(n, g):
    """Row lengths floor(1.55 u^(-1/1.1)) clipped to [1, 4096] (about 9.5 on
    average), columns uniform and distinct, values N(0, 1)."""
    u = 1.0 - torch.rand(n, generator=g, dtype=torch.float64, device=DEV)
    lens = torch.clamp(torch.floor(1.55 * u ** (-1.0 / 1.1)), 1, min(4096, n)).to(torch.int64)
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), lens)
    key = torch.unique(rows * n + torch.randint(0, n, (rows.numel(),), generator=g, device=DEV))   # sorted
    rows = key // n
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(torch.bincount(rows, minlength=n), 0, out=rp[1:])
    val = torch.randn(key.numel(), generator=g, dtype=torch.float64, device=DEV)
    return SimpleNamespace(n=n, rp=rp, col=(key - rows * n).to(torch.int32), val=val)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) + 1)


def _matrix(case, g):
    if case["matrix"] == "powerlaw":
        return _powerlaw_csr(case["nx"], g)
    return _grid_csr(case["matrix"], case["nx"], case["ny"], case["nz"], g, case.get("beta", 0.0))


def _uniform(n, g):
    return 2.0 * torch.rand(n, generator=g, dtype=torch.float64, device=DEV) - 1.0


def _product(A, x):
    rows = torch.repeat_interleave(torch.arange(A.n, device=x.device), torch.diff(A.rp))
    return torch.zeros(A.n, dtype=torch.float64, device=x.device).index_add_(0, rows, A.val * x[A.col.long()])


def _stencil_product(A, x):
    """A x of a grid operator, direction by direction (the same bits every time)."""
    y = torch.zeros_like(x)
    for d in A.dirs:
        y += (A.grid[d] * _shifted(x.reshape(A.grid[d].shape), d)).reshape(-1)
    return y


def _host(A):
    """Host CSR as the package's own containers take it."""
    rp = A.rp.cpu().numpy()
    return SimpleNamespace(n_rows=A.n, n_cols=A.n, nnz=int(rp[-1]), row_ptr=rp, col=A.col.cpu().numpy(),
                           val=A.val.cpu().numpy())


def _vector(t):
    """The package's vector over a torch tensor's memory."""
    return mtl.dense_vector(t.numel(), NUMPY["f64" if t.dtype == torch.float64 else "f32"],
                            _wrap_ptr=t.data_ptr())


def _settle():
    """Waits for torch's stream: the package's context runs on a stream of its own."""
    if DEV.type == "cuda":
        torch.cuda.synchronize()


# ------------------------------------------------------------------ inputs

def _inputs(case, seed):
    """Matrix and vectors of a case in 64 bits."""
    g = _generator(seed)
    A = _matrix(case, g)
    if case["kind"] == "mult":
        x, y0 = _uniform(A.n, g), _uniform(A.n, g)
        return SimpleNamespace(A=A, x=x, y0=y0)
    if case["kind"] == "apply":
        return SimpleNamespace(A=A, x=_uniform(A.n, g))
    x = _uniform(A.n, g)
    return SimpleNamespace(A=A, x=x, b=_stencil_product(A, x))


def _systems(case, seed):
    """The batch's systems: sizes log-uniform, every other one 3D."""
    g, out = _generator(seed), []
    sizes = np.random.default_rng(case["spread"])
    for k in range(case["count"]):
        n = math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))
        three = k % 2 == 1
        m = max(3, int(round(n ** (1.0 / 3.0 if three else 0.5))))
        pc = "diagonal" if sizes.random() < 0.5 else "ic_0"
        A = _grid_csr("grid3d" if three else "grid2d", m, m, m if three else 1, g)
        x = _uniform(A.n, g)
        out.append(SimpleNamespace(A=A, x=x, b=_stencil_product(A, x), pc=pc))
    return out


def prepare(case, seed):
    if case["kind"] == "batch":
        # host arrays: what a program hands to a batch
        s = SimpleNamespace(case=case, systems=[(_host(q.A), q.b.cpu().numpy(), q.pc) for q in _systems(case, seed)])
        return s
    q = _inputs(case, seed)
    h = _host(q.A)
    s = SimpleNamespace(case=case, n=q.A.n)
    if case["kind"] == "mult":
        f32 = case["dtype"] == "f32"
        if case["fmt"] == "csr":
            s.A = mtl.compressed2D.from_problem(h)
        elif case["fmt"] == "ell":
            s.A = mtl.ell_matrix.from_csr(h)
        else:
            s.A = mtl.sparse_banded.from_csr(h)
        s.tx = q.x.to(TORCH[case["dtype"]])
        s.ty = q.y0.to(TORCH[case["dtype"]])
        s.x, s.y = _vector(s.tx), _vector(s.ty)
        if f32 and case["fmt"] == "csr":
            # the FP32 copy of the values is made once, by a matrix's first FP32 product
            t = torch.zeros_like(s.tx)
            _settle()
            mtl.mult(s.A, s.x, _vector(t))
            mtl.default_context().synchronize()
        return s
    s.A = mtl.compressed2D.from_problem(h)
    if case["kind"] == "apply":
        s.P = getattr(itl.pc, case["pc"])(s.A, NUMPY[case["storage"]])
        s.tx = q.x.to(TORCH[case["dtype"]])
        s.ty = torch.zeros_like(s.tx)
        s.x, s.y = _vector(s.tx), _vector(s.ty)
        return s
    if case["kind"] == "solve":
        s.P = getattr(itl.pc, case["pc"])(s.A)
        s.none = itl.pc.identity(s.A)
    s.tb, s.tx = q.b, torch.zeros_like(q.b)
    s.b, s.x = _vector(s.tb), _vector(s.tx)
    return s


# ------------------------------------------------------------------ passes

def run(s):
    case = s.case
    if case["kind"] == "mult":
        mtl.mult(s.A, s.x, s.y, case["assign"])
        return s.ty
    if case["kind"] == "apply":
        itl.solve(s.P, s.x, s.y)
        return s.ty
    if case["kind"] == "solve":
        s.x.fill(0.0)
        it = itl.basic_iteration(s.b, 4000, case["rtol"])
        if case["solver"] == "cg":
            itl.cg(s.A, s.x, s.b, s.P, it)
        elif case["solver"] == "bicgstab":
            itl.bicgstab(s.A, s.x, s.b, s.P, it)
        else:
            itl.gmres(s.A, s.x, s.b, s.P, s.none, it, 30)
        return {"x": s.tx, "iterations": it.iterations(), "error": it.error_code()}
    if case["kind"] == "step":
        s.x.fill(0.0)
        P = getattr(itl.pc, case["pc"])(s.A, np.float32)
        it = itl.refine(case["solver"], s.A, s.x, s.b, P, rtol=case["rtol"])
        return {"x": s.tx, "iterations": it.iterations(), "outer": it.outer, "error": it.error_code()}
    B = serve.batch()
    for A, b, pc in s.systems:
        B.add(A, b, "cg", pc, max_iter=4000, rtol=case["rtol"])
    B.solve(mixed=case["mixed"], rtol=case["rtol"])
    got = [B.result(k) for k in range(len(B))]
    return {"x": [r.x for r in got], "iterations": np.array([r.iterations for r in got])}


# ------------------------------------------------------------------ 64-bit results

def _levels(shape, matrix):
    """Points of each dependency level of a lower sweep (i + j + k, or i + 2 j
    for the 9-point operator), as flat indices into a grid padded by one."""
    nz, ny, nx = shape
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    lev = (i + (2 if matrix == "nine" else 1) * j + k).reshape(-1)
    flat = ((i + 1) + (nx + 2) * ((j + 1) + (ny + 2) * (k + 1))).reshape(-1)
    order = np.argsort(lev, kind="stable")
    cuts = np.cumsum(np.bincount(lev))[:-1]
    return np.split(flat[order], cuts)


def _apply_exact(case, q):
    """ILU(0) / IC(0) of a grid operator and its apply, level by level."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dirs, off = q.A.dirs, {d: d[0] + (nx + 2) * (d[1] + (ny + 2) * d[2]) for d in q.A.dirs}

    def padded(t):
        out = np.zeros((nz + 2, ny + 2, nx + 2))
        out[1:-1, 1:-1, 1:-1] = t.cpu().numpy().reshape(nz, ny, nx)
        return out.reshape(-1)

    a = {d: padded(q.A.grid[d]) for d in dirs}
    centre = (0, 0, 0)
    lower, upper = dirs[:dirs.index(centre)], dirs[dirs.index(centre) + 1:]
    levels = _levels((nz, ny, nx), case["matrix"])
    x = padded(q.x)
    piv = np.zeros_like(x)
    if case["pc"] == "ilu_0":
        for r in levels:
            for d in lower:   # ascending columns
                l = a[d][r] * piv[r + off[d]]
                a[d][r] = l
                for e in dirs[dirs.index(d) + 1:]:
                    w = tuple(p - m for p, m in zip(e, d))   # entry of the neighbour's row in the same column
                    if w in off:
                        a[e][r] -= l * a[w][r + off[d]]
            piv[r] = 1.0 / a[centre][r]
        for r in levels:
            for d in lower:
                x[r] -= a[d][r] * x[r + off[d]]
        for r in reversed(levels):
            for e in upper:
                x[r] -= a[e][r] * x[r + off[e]]
            x[r] *= piv[r]
    else:
        up = {d: a[tuple(-c for c in d)] for d in lower}   # a_ki of the earlier neighbour k in direction d
        for r in levels:
            u = a[centre][r]
            for d in lower:
                u = u - (up[d][r + off[d]] * piv[r + off[d]]) ** 2
            piv[r] = 1.0 / np.sqrt(u)
        for r in levels:
            for d in lower:
                x[r] -= up[d][r + off[d]] * piv[r + off[d]] * x[r + off[d]]
            x[r] *= piv[r]
        for r in reversed(levels):
            for e in upper:
                x[r] -= a[e][r] * piv[r] * x[r + off[e]]
            x[r] *= piv[r]
    return torch.from_numpy(np.ascontiguousarray(x.reshape(nz + 2, ny + 2, nx + 2)[1:-1, 1:-1, 1:-1]).reshape(-1))


def exact(case, seed):
    if case["kind"] == "batch":
        return {"x": [q.x.cpu().numpy() for q in _systems(case, seed)], "iterations": None}
    q = _inputs(case, seed)
    if case["kind"] == "mult":
        x = q.x.to(TORCH[case["dtype"]]).double()
        y = _product(q.A, x)
        return y + q.y0.to(TORCH[case["dtype"]]).double() if case["assign"] == "+=" else y
    if case["kind"] == "apply":
        q.x = q.x.to(TORCH[case["dtype"]]).double()
        return _apply_exact(case, q)
    out = {"x": q.x, "iterations": None, "error": None}   # b = A x
    return dict(out, outer=None) if case["kind"] == "step" else out


# ------------------------------------------------------------------ work

def _entries(case):
    """(rows, entries) of a case's matrix."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["matrix"] == "powerlaw":
        return nx, int(9.5 * nx)
    nnz = 0
    for d in _directions(case["matrix"]):
        nnz += max(nx - abs(d[0]), 0) * max(ny - abs(d[1]), 0) * max(nz - abs(d[2]), 0)
    return nx * ny * nz, nnz


def _solve_work(n, nnz, iters, products, applies, vectors, s):
    """Bytes and operations of `iters` iterations with matrix values of s bytes."""
    product = (s + 4) * nnz + 4 * n + 2 * s * n
    apply_ = s * nnz + s * n + 2 * s * n
    return (iters * (products * product + applies * apply_ + vectors * s * n),
            iters * (2 * products * nnz + 2 * applies * nnz + 2 * vectors * n))


def _iterations(pc, side, solver):
    """About what these operators take to 1e-8 (for the estimate of the work only)."""
    per = {"diagonal": 2.2, "ic_0": 0.7, "ilu_0": 0.5}[pc] * (1.0 if solver == "cg" else 0.9)
    return max(5.0, per * side)


def work(case):
    if case["kind"] == "batch":
        sizes, b, f = np.random.default_rng(case["spread"]), 0.0, 0.0
        for k in range(case["count"]):
            n = math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))
            pc = "diagonal" if sizes.random() < 0.5 else "ic_0"
            d = 3 if k % 2 == 1 else 2
            w = _solve_work(n, (2 * d + 1) * n, _iterations(pc, n ** (1.0 / d), "cg"), 1, int(pc == "ic_0"), 6, 8)
            b, f = b + w[0], f + w[1]
        return {"bytes": b, "flops": f}
    n, nnz = _entries(case)
    if case["kind"] == "mult":
        s = 8 if case["dtype"] == "f64" else 4
        idx = {"csr": 4 * nnz + 4 * (n + 1), "ell": 4 * nnz, "banded": 0}[case["fmt"]]
        return {"bytes": s * nnz + idx + s * n * (3 if case["assign"] == "+=" else 2), "flops": 2 * nnz}
    if case["kind"] == "apply":
        st, sv = (8 if case[k] == "f64" else 4 for k in ("storage", "dtype"))
        return {"bytes": st * nnz + st * n * (case["pc"] == "ic_0") + 2 * sv * n, "flops": 2 * nnz}
    side = max(case["nx"], case["ny"], case["nz"])
    it = _iterations(case["pc"], side, case["solver"])
    products, vectors = {"cg": (1, 6), "bicgstab": (2, 12), "gmres": (1, 34)}[case["solver"]]
    applies = products if case["pc"] != "diagonal" else 0
    b, f = _solve_work(n, nnz, it, products, applies, vectors, 4 if case["kind"] == "step" else 8)
    if case["kind"] == "step":
        b += 12 * nnz + 8 * nnz   # set-up: the matrix read, the factors written once
    return {"bytes": b, "flops": f}
