"""CG and BiCGStab in FP32 and FP64 on the loops that their sizes choose (one
cooperative kernel with one to four rows per thread, split passes with one
column or column slices, short rows and longer ones, dots fused or apart), with
scalar and block Jacobi: columns that stop at different iterations, checked
on the FP64 residual; and a solve that outlasts one launch of the cooperative
kernel."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Bicgstab, Cg, Iteration, Jacobi, ResidualNorm

pytestmark = pytest.mark.gpu

EPS = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24}


def banded(n, band, symmetric):
    """Strictly dominant: 2 * band + 1 entries per inner row, the diagonal
    between 4 band and 4 band + 2, the others at most 1."""
    rng = np.random.default_rng(n)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [4.0 * band + rng.uniform(0, 2, n)]
    for d in range(1, min(band, n - 1) + 1):
        up = -rng.uniform(0.5, 1.0, n - d)
        i = np.arange(n - d)
        rows += [i, i + d]
        cols += [i + d, i]
        vals += [up, up if symmetric else rng.uniform(-1.0, 0.5, n - d)]
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), cols[o].astype(np.int32), vals[o]


def product(rp, ci, v, x):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    return np.stack([np.bincount(rows, weights=v * c[ci], minlength=len(rp) - 1) for c in x.T], 1)


def check(factory, symmetric, n, band, k, dt, block):
    exe = CudaExecutor.create(0)
    rp, ci, v = banded(n, band, symmetric)
    A = Csr.read(exe, rp, ci, v, dtype=dt)
    v = A.values.double().cpu().numpy()
    rng = np.random.default_rng(k)
    x0 = torch.from_numpy(rng.standard_normal((n, k))).to(dt)
    b = rng.standard_normal((n, k))
    if k > 1:
        b[:, 0] = product(rp, ci, v, x0.double().numpy()[:, :1])[:, 0]  # starts near the solution
        b[:, 1] = b[:, 0] + 1e-3 * rng.standard_normal(n)               # stops early
    b = torch.from_numpy(b).to(dt)
    tol, its = (1e-11, 80) if dt == torch.float64 else (1e-5, 40)
    s = (factory.build().with_criteria(Iteration.build().with_max_iters(its),
                                       ResidualNorm.build().with_reduction_factor(tol))
         .with_preconditioner(Jacobi.build().with_max_block_size(block)).on(exe).generate(A))
    wide = torch.full((n, k + 1), 7.0, dtype=dt, device="cuda")
    x = wide[:, :k]
    x.copy_(x0)
    s.apply(b.cuda(), x)
    # condition below 3 (dominance by a half): about 2 digits per 4 iterations
    assert s.logger.num_iterations < its and s.logger.has_converged
    got, bh = x.double().cpu().numpy(), b.double().numpy()
    res = np.linalg.norm(bh - product(rp, ci, v, got), axis=0)
    # the recursive residual meets tol ||b||; each iteration's updates of x
    # and r and its product (2 band + 1 terms) round within (2 band + 5) eps
    # of ||A|| ||x||, ||A|| <= 6 band + 2, over at most `its` iterations, for
    # iterates up to the larger of x0 and the solution
    size = np.linalg.norm(got, axis=0) + np.linalg.norm(x0.double().numpy(), axis=0)
    allow = tol * np.linalg.norm(bh, axis=0) + \
        its * (2 * band + 5) * EPS[dt] * (6 * band + 2) * size
    assert np.all(res <= allow), (res / allow)
    assert bool((wide[:, k] == 7.0).all())


TYPES = pytest.mark.parametrize("dt", [torch.float64, torch.float32])


@TYPES
@pytest.mark.parametrize("n,band,k", [(75776, 1, 1), (75777, 1, 1), (151553, 1, 1),
                                      (303104, 1, 1), (303105, 1, 1), (131072, 30, 1),
                                      (49153, 1, 8), (98305, 3, 8), (6200, 13, 8), (24577, 1, 16),
                                      (3100, 13, 16), (98304, 1, 4), (12289, 6, 4)])
def test_cg(n, band, k, dt):
    check(Cg, True, n, band, k, dt, 1)


@TYPES
@pytest.mark.parametrize("n,band,k", [(524287, 1, 1), (524288, 1, 1), (600001, 2, 1), (5001, 2, 2),
                                      (40000, 5, 2), (5001, 2, 4), (700, 40, 4), (196607, 6, 4),
                                      (196608, 6, 4), (9000, 3, 8), (4099, 6, 16), (700, 40, 16)])
def test_bicgstab(n, band, k, dt):
    check(Bicgstab, False, n, band, k, dt, 1)


@TYPES
@pytest.mark.parametrize("block", [2, 8, 16, 32])
@pytest.mark.parametrize("n,band,k", [(131073, 1, 1), (98305, 1, 4), (49153, 2, 8), (24577, 1, 16),
                                      (12289, 6, 4), (3100, 13, 16)])
def test_block_jacobi(n, band, k, block, dt):
    check(Cg, True, n, band, k, dt, block)
    if n < 50000:
        check(Bicgstab, False, n, band, k, dt, block)


def test_solve_longer_than_a_launch():
    """tridiag(-1, 2, -1) x = 1 takes n / 2 iterations: the directions are
    exact in FP64 (x_i = i (n + 1 - i) / 2 exactly in numpy), and 10,000
    iterations cross a launch of 8,192."""
    n = 20000
    rows = np.arange(n)
    cols = np.stack([rows - 1, rows, rows + 1], 1)
    ok = (cols >= 0) & (cols < n)
    v = np.broadcast_to([-1.0, 2.0, -1.0], cols.shape)[ok]
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))])
    exe = CudaExecutor.create(0)
    A = Csr.read(exe, rp.astype(np.int32), cols[ok].astype(np.int32), v)
    s = (Cg.build().with_criteria(Iteration.build().with_max_iters(12000),
                                  ResidualNorm.build().with_reduction_factor(1e-10))
         .with_preconditioner(Jacobi.build().with_max_block_size(1)).on(exe).generate(A))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    s.apply(torch.ones(n, dtype=torch.float64, device="cuda"), x)
    assert s.logger.num_iterations == n // 2 and s.logger.has_converged
    i = np.arange(1, n + 1)
    ref = i * (n + 1.0 - i) / 2
    assert np.abs(x.cpu().numpy() - ref).max() <= 1e-9 * ref.max()
