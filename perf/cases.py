"""Performance cases: what a user of this package has it do, through its
public entry points.

Four kinds, each a plain dict:

- "spmv": one product of a sparse matrix with a block of vectors, in every
  format (Csr classical and load_balance, Ell, Sellp), FP64 and FP32, one to
  sixteen columns, plain (x = A b) or as the residual r = b - A x.
- "solve": one linear solve with CG, BiCGStab, GMRES or mixed-precision
  iterative refinement (IR) and scalar Jacobi, to a tolerance or for a fixed
  number of iterations.
- "batch": BiCGStab on thousands of small independent systems.
- "autograd": a differentiable solve, forward and backward.

Matrices are the package's own workloads (2D 5-point and 3D 7-point Poisson,
3D 27-point anisotropic diffusion, 2D convection-diffusion, variable
conductivity, random power-law rows), assembled here on the GPU.  `exact`
restates each computation in plain FP64 torch.
"""
import itertools
import math

import numpy as np
import torch

from ginkgo_b200.autograd import ConductivityOperator
from ginkgo_b200.batch import BatchBicgstab, BatchEll
from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Bicgstab, Cg, Gmres, Ir, Iteration, Jacobi, ResidualNorm
from ginkgo_b200.stencils import conductivity_edges

DTYPES = {"f64": torch.float64, "f32": torch.float32}
L2_BYTES = 126 << 20


def listed():
    return [
        # the smallest calls: one product with the 65,536-row system, as an
        # outer iteration or a time stepper issues it; launch and latency
        {"name": "spmv_csr_2d256", "kind": "spmv", "matrix": "2d5", "nx": 256, "format": "csr",
         "dtype": "f64", "k": 1, "residual": False},
        # the headline product: 14.6M entries, streamed from HBM
        {"name": "spmv_csr_3d128", "kind": "spmv", "matrix": "3d7", "nx": 128, "format": "csr",
         "dtype": "f64", "k": 1, "residual": False},
        # graph-like rows of very uneven length, what load_balance is for
        {"name": "spmv_lb_powerlaw", "kind": "spmv", "matrix": "powerlaw", "nx": 1000003,
         "format": "load_balance", "dtype": "f64", "k": 1, "residual": False},
        # block products (block Krylov methods, several load cases)
        {"name": "spmv_sellp_3d128_k16", "kind": "spmv", "matrix": "3d7", "nx": 128,
         "format": "sellp", "dtype": "f64", "k": 16, "residual": False},
        # residuals of four FP32 columns on an odd-sized 27-point grid
        {"name": "spmv_ell_27pt_f32_k4", "kind": "spmv", "matrix": "3d27", "nx": 77,
         "format": "ell", "dtype": "f32", "k": 4, "residual": True},
        # a whole small solve to 1e-10 (710 iterations): launches and latency
        {"name": "cg_2d256", "kind": "solve", "solver": "cg", "matrix": "2d5", "nx": 256, "k": 1,
         "max_iters": 1000, "tol": 1e-10, "krylov_dim": 0},
        # a large system, iterations bound by memory
        {"name": "cg_3d128", "kind": "solve", "solver": "cg", "matrix": "3d7", "nx": 128, "k": 1,
         "max_iters": 40, "tol": 1e-10, "krylov_dim": 0},
        # an implicit time step of a convection-diffusion system with several
        # right-hand sides
        {"name": "bicgstab_cd700_k4", "kind": "solve", "solver": "bicgstab", "matrix": "cd2d",
         "nx": 700, "k": 4, "max_iters": 100, "tol": 1e-10, "krylov_dim": 0},
        # restarted FP64 GMRES, the baseline of mixed precision
        {"name": "gmres30_27pt96", "kind": "solve", "solver": "gmres", "matrix": "3d27", "nx": 96,
         "k": 1, "max_iters": 150, "tol": 1e-10, "krylov_dim": 30},
        # the mixed-precision solve to 1e-10: FP32 GMRES(30) inside FP64
        # refinement
        {"name": "ir_f32_27pt96", "kind": "solve", "solver": "ir", "matrix": "3d27", "nx": 96,
         "k": 1, "max_iters": 5000, "tol": 1e-10, "krylov_dim": 30},
        # thousands of small ragged systems (implicit chemistry, cell-wise
        # transport), 32 to 1024 rows each
        {"name": "batch_bicgstab_8192", "kind": "batch", "systems": 8192, "lo": 32, "hi": 1024,
         "tol": 1e-8, "max_iters": 500, "sizes_seed": 0},
        # training through a PDE solve: 16 load cases, gradient to the
        # conductivities
        {"name": "autograd_64_k16", "kind": "autograd", "nx": 64, "k": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "solve", "solve", "batch", "autograd"])
    if kind == "spmv":
        matrix = rng.choice(["2d5", "3d7", "3d27", "powerlaw"])
        fmt = rng.choice(["csr", "load_balance", "sellp"] if matrix == "powerlaw"
                         else ["csr", "load_balance", "ell", "sellp"])
        nx = {"2d5": lambda: _log_int(rng, 64, 1400), "3d7": lambda: _log_int(rng, 16, 128),
              "3d27": lambda: _log_int(rng, 16, 96),
              "powerlaw": lambda: _log_int(rng, 20000, 1000000)}[matrix]()
        return {"kind": "spmv", "matrix": matrix, "nx": nx, "format": fmt,
                "dtype": rng.choice(["f64", "f64", "f32"]), "k": rng.choice([1, 1, 2, 3, 4, 8, 16]),
                "residual": rng.random() < 0.3}
    if kind == "solve":
        solver = rng.choice(["cg", "cg", "bicgstab", "gmres", "ir"])
        c = {"kind": "solve", "solver": solver, "k": 1, "tol": 1e-10, "krylov_dim": 0}
        if solver == "cg":
            c["matrix"] = rng.choice(["2d5", "3d7"])
            c["nx"] = _log_int(rng, 64, 1000) if c["matrix"] == "2d5" else _log_int(rng, 20, 128)
            c["k"] = rng.choice([1, 1, 4, 16])
            c["max_iters"] = rng.randint(20, 60)
        elif solver == "bicgstab":
            c["matrix"] = "cd2d"
            c["nx"] = _log_int(rng, 64, 1000)
            c["k"] = rng.choice([1, 1, 4])
            c["max_iters"] = 100
        else:
            c["matrix"] = "3d27"
            c["nx"] = _log_int(rng, 16, 80)
            c["krylov_dim"] = rng.choice([20, 30, 50])
            c["max_iters"] = rng.randint(40, 150) if solver == "gmres" else 5000
        return c
    if kind == "batch":
        lo = rng.choice([16, 32, 64])
        return {"kind": "batch", "systems": _log_int(rng, 200, 8000), "lo": lo,
                "hi": rng.randint(4 * lo, 1024), "tol": 1e-8, "max_iters": 500,
                "sizes_seed": rng.randint(1, 10 ** 6)}
    return {"kind": "autograd", "nx": _log_int(rng, 12, 63), "k": rng.choice([1, 4, 16])}


# ------------------------------------------------------------ matrices --
def _grid(nx, dim, offsets, weights, dtype):
    """Csr arrays of a constant stencil on an nx^dim grid, Dirichlet boundary
    eliminated; offsets are (x, y[, z]) tuples."""
    n = nx ** dim
    shifts = [sum(o * nx ** a for a, o in enumerate(off)) for off in offsets]
    order = sorted(range(len(offsets)), key=shifts.__getitem__)
    idx = torch.arange(n, device="cuda")
    xyz = [(idx // nx ** a) % nx for a in range(dim)]
    ok = torch.ones(n, len(offsets), dtype=torch.bool, device="cuda")
    for j, s in enumerate(order):
        for a, o in enumerate(offsets[s]):
            if o:
                ok[:, j] &= (xyz[a] + o >= 0) & (xyz[a] + o < nx)
    cols = idx[:, None] + torch.tensor([shifts[s] for s in order], device="cuda")
    w = torch.tensor([weights[s] for s in order], dtype=torch.float64, device="cuda")
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(ok.sum(1), 0, out=rp[1:])
    return n, rp.int(), cols[ok].int(), w.expand(n, -1)[ok].to(dtype)


def _axis_offsets(dim):
    return [(0,) * dim] + [tuple(s * (a == b) for b in range(dim)) for a in range(dim)
                           for s in (1, -1)]


def _matrix(case, seed, dtype):
    """(n, row_ptrs, col_idxs, values) on the GPU."""
    kind, nx = case["matrix"], case["nx"]
    if kind == "2d5":
        return _grid(nx, 2, _axis_offsets(2), [4.0] + [-1.0] * 4, dtype)
    if kind == "3d7":
        return _grid(nx, 3, _axis_offsets(3), [6.0] + [-1.0] * 6, dtype)
    if kind == "cd2d":
        # one implicit Euler step of 5-point convection-diffusion (identity
        # plus central differences), the diffusion and the velocity drawn per
        # seed
        rng = np.random.default_rng(seed)
        d, (vx, vy) = rng.uniform(0.5, 2.0), rng.uniform(-1.0, 1.0, 2)
        return _grid(nx, 2, _axis_offsets(2),
                     [1 + 4 * d, -d + vx / 2, -d - vx / 2, -d + vy / 2, -d - vy / 2], dtype)
    if kind == "3d27":
        S, M = {-1: -1.0, 0: 2.0, 1: -1.0}, {-1: 1 / 6, 0: 2 / 3, 1: 1 / 6}
        offs = list(itertools.product((-1, 0, 1), repeat=3))
        ws = [S[x] * M[y] * M[z] + 1e-2 * M[x] * S[y] * M[z] + 1e-4 * M[x] * M[y] * S[z]
              for x, y, z in offs]
        return _grid(nx, 3, offs, ws, dtype)
    # power law: row lengths lognormal(2.5, 1) in [1, 4096], uniform columns
    # without duplicates, N(0, 1) values; the pattern belongs to the size
    n = nx
    g = torch.Generator("cuda").manual_seed(n)
    lens = torch.empty(n, dtype=torch.float64, device="cuda").normal_(2.5, 1.0, generator=g)
    lens = lens.exp().round().clamp(1, min(4096, n)).long()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    cols = torch.randint(n, rows.shape, device="cuda", generator=g)
    key = torch.unique(rows * n + cols)
    rows, cols = key // n, key % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(rows, minlength=n), 0, out=rp[1:])
    g.manual_seed(seed)
    v = torch.randn(cols.shape, dtype=torch.float64, device="cuda", generator=g)
    return n, rp.int(), cols.int(), v.to(dtype)


def _counts(case):
    """(rows, stored entries) of the Csr matrix of a case, for work()."""
    nx = case["nx"]
    return {"2d5": lambda: (nx ** 2, 5 * nx ** 2 - 4 * nx),
            "cd2d": lambda: (nx ** 2, 5 * nx ** 2 - 4 * nx),
            "3d7": lambda: (nx ** 3, 7 * nx ** 3 - 6 * nx ** 2),
            "3d27": lambda: (nx ** 3, (3 * nx - 2) ** 3),
            # mean of round(lognormal(2.5, 1))
            "powerlaw": lambda: (nx, int(20.1 * nx))}[case["matrix"]]()


def _vectors(n, k, seed, dtype, uniform=False):
    g = torch.Generator("cuda").manual_seed(1000003 + seed)
    t = torch.empty((n, k) if k > 1 else (n,), dtype=torch.float64, device="cuda")
    t = t.uniform_(-1, 1, generator=g) if uniform else t.normal_(generator=g)
    return t.to(dtype)


# --------------------------------------------------------------- batch --
def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes_seed"])
    return rng.integers(case["lo"], case["hi"] + 1, size=case["systems"])


def _batch_system(case, seed):
    """Ragged batch of 5-point convection-diffusion systems on the
    most-square grids of their sizes: (row offsets, col_idxs, values), five
    column-major entries per row, padding column -1."""
    sizes = _batch_sizes(case)
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.5, 2.0, len(sizes))
    vel = rng.uniform(-1.0, 1.0, (len(sizes), 2))
    ny = np.array([max(a for a in range(1, math.isqrt(int(s)) + 1) if s % a == 0) for s in sizes])
    offs = np.zeros(len(sizes) + 1, dtype=np.int64)
    np.cumsum(sizes, out=offs[1:])
    per_row = lambda a: torch.from_numpy(np.repeat(a, sizes)).cuda()  # noqa: E731
    start, n, nx = per_row(offs[:-1]), per_row(sizes), per_row(sizes // ny)
    r = torch.arange(int(offs[-1]), device="cuda") - start
    x, dd, vx, vy = r % nx, per_row(d), per_row(vel[:, 0]), per_row(vel[:, 1])
    one = torch.ones_like(nx)
    # south, west, diagonal, east, north: ascending columns
    parts = [(-nx, r - nx >= 0, -dd - vy / 2), (-one, x > 0, -dd - vx / 2), (0 * one, n > 0, 4 * dd),
             (one, x < nx - 1, -dd + vx / 2), (nx, r + nx < n, -dd + vy / 2)]
    ci = torch.full((5 * len(r),), -1, dtype=torch.int32, device="cuda")
    v = torch.zeros(5 * len(r), dtype=torch.float64, device="cuda")
    slot = torch.zeros_like(r)
    for shift, ok, w in parts:  # the present neighbours fill the row's slots in turn
        at = (5 * start + slot * n + r)[ok]
        ci[at] = (r + shift)[ok].int()
        v[at] = w[ok]
        slot += ok
    return offs, ci, v


# ------------------------------------------------------------- measured --
def prepare(case, seed):
    exe = CudaExecutor.create(0)
    if case["kind"] == "spmv":
        dtype = DTYPES[case["dtype"]]
        n, rp, ci, v = _matrix(case, seed, dtype)
        fmt = case["format"]
        A = Csr(exe, (n, n), rp, ci, v, "load_balance" if fmt == "load_balance" else "classical")
        A = A.convert_to_ell() if fmt == "ell" else A.convert_to_sellp(32) if fmt == "sellp" else A
        x = _vectors(n, case["k"], seed, dtype)
        s = {"A": A, "x": x, "y": torch.empty_like(x)}
        if case["residual"]:
            s["b"] = _vectors(n, case["k"], seed + 7, dtype)
            s["one"] = torch.ones(1, dtype=dtype, device="cuda")
            s["minus_one"] = -s["one"]
        return s
    if case["kind"] == "solve":
        n, rp, ci, v = _matrix(case, seed, torch.float64)
        A = Csr(exe, (n, n), rp, ci, v)
        x_true = _vectors(n, case["k"], seed, torch.float64, uniform=True)
        b = torch.empty_like(x_true)
        A.apply(x_true, b)
        crit = (Iteration.build().with_max_iters(case["max_iters"]),
                ResidualNorm.build().with_reduction_factor(case["tol"]))
        jacobi = Jacobi.build().with_max_block_size(1)
        if case["solver"] == "ir":
            inner = (Gmres.build().with_krylov_dim(case["krylov_dim"])
                     .with_storage_precision("f32").with_preconditioner(jacobi))
            f = Ir.build().with_solver(inner).with_criteria(*crit)
        else:
            f = {"cg": Cg, "bicgstab": Bicgstab, "gmres": Gmres}[case["solver"]].build()
            f = f.with_criteria(*crit).with_preconditioner(jacobi)
            if case["solver"] == "gmres":
                f = f.with_krylov_dim(case["krylov_dim"])
        return {"solver": f.on(exe).generate(A), "b": b, "x": torch.zeros_like(b)}
    if case["kind"] == "batch":
        offs, ci, v = _batch_system(case, seed)
        A = BatchEll(exe, offs, 5, ci, v)
        f = (BatchBicgstab.build().with_max_iterations(case["max_iters"])
             .with_tolerance(case["tol"]).with_tolerance_type("relative")
             .with_preconditioner("jacobi"))
        b = _vectors(int(offs[-1]), 1, seed, torch.float64)
        return {"solver": f.on(exe).generate(A), "b": b, "x": torch.zeros_like(b)}
    op = ConductivityOperator(case["nx"])
    g = torch.Generator("cuda").manual_seed(seed)
    theta = torch.empty(op.num_edges, dtype=torch.float64, device="cuda")
    theta = theta.log_normal_(0.0, 0.5, generator=g).requires_grad_()
    b = _vectors(op.n, case["k"], seed, torch.float64).requires_grad_()
    return {"op": op, "theta": theta, "b": b,
            "target": _vectors(op.n, case["k"], seed + 7, torch.float64)}


def run(state):
    if "A" in state:
        if "b" in state:  # r = b - A x
            state["y"].copy_(state["b"])
            return state["A"].apply(state["minus_one"], state["x"], state["one"], state["y"])
        return state["A"].apply(state["x"], state["y"])
    if "solver" in state:
        state["x"].zero_()
        return state["solver"].apply(state["b"], state["x"])
    x = state["op"].solve(state["theta"], state["b"])
    loss = (x - state["target"]).square().sum()
    d_theta, d_b = torch.autograd.grad(loss, (state["theta"], state["b"]))
    return {"x": x.detach(), "d_theta": d_theta, "d_b": d_b}


def work(case):
    """The matrix and every vector block once per product; a solve reads a
    matrix (and a Krylov basis) that does not fit the L2 cache in every
    iteration, a smaller one once."""
    if case["kind"] == "spmv":
        n, nnz = _counts(case)
        s, k = 8 if case["dtype"] == "f64" else 4, case["k"]
        return {"bytes": nnz * (s + 4) + 4 * (n + 1) + (3 if case["residual"] else 2) * n * k * s,
                "flops": 2 * nnz * k}
    if case["kind"] == "solve":
        n, nnz = _counts(case)
        k, its = case["k"], case["max_iters"]
        if its >= 100 and case["solver"] != "gmres":
            # to the tolerance: about 28 iterations on a time step, otherwise
            # in proportion to the grid
            its = {"bicgstab": 28, "cg": 2.8 * case["nx"], "ir": 13 * case["nx"]}[case["solver"]]
        a = nnz * (8 if case["solver"] == "ir" else 12) + 4 * n
        per = {"cg": 1, "bicgstab": 2}.get(case["solver"], 1)
        basis = 0.5 * case["krylov_dim"] * n * (4 if case["solver"] == "ir" else 8)
        big = its if a > L2_BYTES else 1
        return {"bytes": per * big * a + (its * basis if 2 * basis > L2_BYTES else 2 * basis)
                + 2 * n * k * 8,
                "flops": its * (per * 2 * nnz * k + 10 * n * k + 8 * basis / 8)}
    if case["kind"] == "batch":
        rows = int(_batch_sizes(case).sum())
        return {"bytes": rows * (5 * 12 + 3 * 8), "flops": 34 * rows * 40}
    n, k = case["nx"] ** 3, case["k"]
    its = int(4.5 * case["nx"])
    return {"bytes": 7 * n * 12 + 4 * n * k * 8 + 7 * n * 8, "flops": 2 * its * (14 + 10) * n * k}


# ---------------------------------------------------------------- exact --
def _op(n, rp, ci, v):
    m = torch.sparse_csr_tensor(rp, ci, v.double(), (n, n))
    return lambda x: m @ x


def _rows(n, rp):
    return torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())


def _diagonal(n, rp, ci, v):
    rows = _rows(n, rp)
    on = rows == ci
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_put((rows[on],), v[on].double())


def _dot(a, b):
    return (a * b).sum(0)


def _cg(A, dinv, b, max_iters, tol):
    """Jacobi-preconditioned CG from zero; a column that has met the
    tolerance stays as it is."""
    x, r, p = torch.zeros_like(b), b.clone(), torch.zeros_like(b)
    goal, rho_old = tol * b.norm(dim=0), torch.ones_like(b[0])
    for _ in range(max_iters):
        on = r.norm(dim=0) > goal
        if not bool(on.any()):
            break
        z = dinv * r
        rho = _dot(r, z)
        p = z + rho / rho_old * p
        q = A(p)
        a = torch.where(on, rho / _dot(p, q), 0.0)
        x += a * p
        r -= a * q
        rho_old = rho
    return x


def _bicgstab(A, dinv, b, max_iters, tol):
    x, r, goal = torch.zeros_like(b), b.clone(), tol * b.norm(dim=0)
    rt, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho_old = alpha = omega = torch.ones_like(b[0])
    for _ in range(max_iters):
        on = r.norm(dim=0) > goal
        if not bool(on.any()):
            break
        rho = _dot(rt, r)
        p = r + rho / rho_old * (alpha / omega) * (p - omega * v)
        y = dinv * p
        v = A(y)
        alpha = rho / _dot(rt, v)
        s = r - alpha * v
        z = dinv * s
        t = A(z)
        omega = _dot(s, t) / _dot(t, t)
        x += torch.where(on, alpha * y + omega * z, 0.0)
        r = torch.where(on, s - omega * t, r)
        rho_old = rho
    return x


def _gmres(A, dinv, b, max_iters, tol, dim):
    """Right-preconditioned restarted GMRES for one column."""
    x, goal, left = torch.zeros_like(b), tol * b.norm(), max_iters
    while left > 0:
        r = b - A(x)
        beta = r.norm()
        if beta <= goal:
            break
        V = torch.zeros(dim + 1, len(b), dtype=b.dtype, device=b.device)
        H = torch.zeros(dim + 1, dim, dtype=b.dtype, device=b.device)
        V[0] = r[:, 0] / beta
        for j in range(min(dim, left)):
            w = A(dinv * V[j][:, None])[:, 0]
            for _ in range(2):
                h = V[:j + 1] @ w
                w = w - h @ V[:j + 1]
                H[:j + 1, j] += h
            H[j + 1, j] = w.norm()
            V[j + 1] = w / H[j + 1, j]
            e = torch.zeros(j + 2, 1, dtype=b.dtype, device=b.device)
            e[0] = beta
            y = torch.linalg.lstsq(H[:j + 2, :j + 1], e).solution
            left -= 1
            if (H[:j + 2, :j + 1] @ y - e).norm() <= goal:
                break
        x = x + dinv * (y.T @ V[:j + 1]).T
    return x


def exact(case, seed):
    if case["kind"] == "spmv":
        dtype = DTYPES[case["dtype"]]
        n, rp, ci, v = _matrix(case, seed, dtype)
        y = _op(n, rp, ci, v)(_vectors(n, case["k"], seed, dtype).double())
        return _vectors(n, case["k"], seed + 7, dtype).double() - y if case["residual"] else y
    if case["kind"] == "solve":
        n, rp, ci, v = _matrix(case, seed, torch.float64)
        A, dinv = _op(n, rp, ci, v), 1 / _diagonal(n, rp, ci, v)[:, None]
        x_true = _vectors(n, case["k"], seed, torch.float64, uniform=True)
        b = A(x_true.reshape(n, -1))
        its, tol = case["max_iters"], case["tol"]
        if case["solver"] == "cg":
            x = _cg(A, dinv, b, its, tol)
        elif case["solver"] == "bicgstab":
            x = _bicgstab(A, dinv, b, its, tol)
        elif case["solver"] == "gmres":
            x = _gmres(A, dinv, b, its, tol, case["krylov_dim"])
        else:  # iterative refinement ends near the solution
            x = x_true
        return x.reshape(x_true.shape)
    if case["kind"] == "batch":
        offs, ci, v = _batch_system(case, seed)
        b = _vectors(int(offs[-1]), 1, seed, torch.float64)
        x, sizes = torch.empty_like(b), np.diff(offs)
        order = np.argsort(sizes, kind="stable")
        for part in np.array_split(order, max(1, len(order) // 256)):
            m = int(sizes[part].max())
            D = torch.eye(m, dtype=torch.float64, device="cuda").repeat(len(part), 1, 1)
            R = torch.zeros(len(part), m, 1, dtype=torch.float64, device="cuda")
            for i, s in enumerate(part):
                o, n = int(offs[s]), int(sizes[s])
                c, w = ci[5 * o:5 * (o + n)].long(), v[5 * o:5 * (o + n)]
                rows = torch.arange(5 * n, device="cuda") % n
                block = torch.zeros(n, n + 1, dtype=torch.float64, device="cuda")
                block[rows, c] = w  # padding lands in the last column
                D[i, :n, :n] = block[:, :n]
                R[i, :n, 0] = b[o:o + n]
            sol = torch.linalg.solve(D, R)
            for i, s in enumerate(part):
                o, n = int(offs[s]), int(sizes[s])
                x[o:o + n] = sol[i, :n, 0]
        return x
    s = prepare(case, seed)
    op, theta, n, k = s["op"], s["theta"].detach(), s["op"].n, case["k"]
    b, target = s["b"].detach().reshape(n, k), s["target"].reshape(n, k)
    v = op.values(theta)
    A, dinv = _op(n, op.row_ptrs, op.col_idxs, v), 1 / _diagonal(n, op.row_ptrs, op.col_idxs, v)[:, None]
    x = _cg(A, dinv, b, 2000, 1e-14)
    lam = _cg(A, dinv, 2 * (x - target), 2000, 1e-14)
    # A = sum over edges of theta_e (e_i - e_j)(e_i - e_j)^T, so
    # dL/dtheta_e = -(lam_i - lam_j) . (x_i - x_j), the boundary value being 0
    ei, ej = (torch.from_numpy(t).cuda() for t in conductivity_edges(case["nx"]))
    inner = (ej >= 0).double()[:, None]
    dl = lam[ei] - inner * lam[ej.clamp(min=0)]
    dx = x[ei] - inner * x[ej.clamp(min=0)]
    shape = s["b"].shape
    return {"x": x.reshape(shape), "d_theta": -(dl * dx).sum(1), "d_b": lam.reshape(shape)}
