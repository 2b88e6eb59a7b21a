"""BiCGStab's split iterations with the dots taken inside the SpMVs: one
column of a large system, column slices with short rows (fused) and rows over
64 entries (dots in a pass of their own), columns that stop at different
iterations, against FP64 BiCGStab restated in numpy."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Bicgstab, Iteration, Jacobi, ResidualNorm

pytestmark = pytest.mark.gpu


def banded(n, band, seed):
    """Nonsymmetric, strictly dominant: 2 * band + 1 entries per inner row."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [4.0 * band + rng.uniform(0, 2, n)]
    for d in range(1, min(band, n - 1) + 1):
        i = np.arange(n - d)
        rows += [i, i + d]
        cols += [i + d, i]
        vals += [-rng.uniform(0.5, 1.0, n - d), rng.uniform(-1.0, 0.5, n - d)]
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), cols[o].astype(np.int32), vals[o]


def product(rp, ci, v, x):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    return np.bincount(rows, weights=v * x[ci], minlength=len(rp) - 1)


def bicgstab(rp, ci, v, b, x, its, tol):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    d = 1.0 / v[rows == ci]
    goal = tol * np.linalg.norm(b)
    x, r = x.copy(), b - product(rp, ci, v, x)
    rt, p, q = r.copy(), np.zeros_like(b), np.zeros_like(b)
    rho_old = alpha = omega = 1.0
    for _ in range(its):
        if np.linalg.norm(r) <= goal:
            break
        rho = rt @ r
        p = r + rho / rho_old * alpha / omega * (p - omega * q)
        y = d * p
        q = product(rp, ci, v, y)
        alpha = rho / (rt @ q)
        s = r - alpha * q
        if np.linalg.norm(s) <= goal:
            x += alpha * y
            break
        z = d * s
        t = product(rp, ci, v, z)
        omega = (s @ t) / (t @ t)
        x += alpha * y + omega * z
        r = s - omega * t
        rho_old = rho
    return x


@pytest.mark.parametrize("n,band,k", [(600000, 1, 1), (524288, 2, 1), (1, 1, 4), (33, 1, 4),
                                      (5001, 2, 4), (4099, 6, 16), (700, 40, 8), (20001, 1, 16),
                                      (9000, 3, 3)])
@pytest.mark.parametrize("its", [1, 2, 100])
def test_split_iterations(n, band, k, its):
    exe = CudaExecutor.create(0)
    rp, ci, v = banded(n, band, n)
    rng = np.random.default_rng(k)
    b, x0 = rng.standard_normal((n, k)), rng.standard_normal((n, k))
    if k > 1:
        b[:, 0] = product(rp, ci, v, x0[:, 0])  # starts at the solution
        b[:, 1] = product(rp, ci, v, x0[:, 1] + 1e-6 * rng.standard_normal(n))  # stops early
    x = torch.from_numpy(x0).cuda()
    s = (Bicgstab.build().with_criteria(Iteration.build().with_max_iters(its),
                                        ResidualNorm.build().with_reduction_factor(1e-12))
         .with_preconditioner(Jacobi.build().with_max_block_size(1)).on(exe)
         .generate(Csr.read(exe, rp, ci, v)))
    s.apply(torch.from_numpy(b).cuda(), x)
    got = x.cpu().numpy()
    for j in range(k):
        ref = bicgstab(rp, ci, v, b[:, j], x0[:, j], its, 1e-12)
        # dominant rows (condition below 10): within the tolerance at the end,
        # a few eps per iteration before
        assert np.linalg.norm(got[:, j] - ref) <= 1e-10 * np.linalg.norm(ref), j
