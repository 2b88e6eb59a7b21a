"""CG at the edges of its three loops: the resident kernel (rows per block
and thread, lanes per row, the last size it takes), the split passes (x
applied one pass late, columns that stop at different iterations, strided x)
and the fused passes, against FP64 CG restated in numpy."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Cg, Iteration, Jacobi, ResidualNorm

pytestmark = pytest.mark.gpu


def banded(n, band, seed):
    """Symmetric, strictly dominant: 2 * band + 1 entries per inner row."""
    rng = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [4.0 * band + rng.uniform(0, 2, n)]
    for d in range(1, min(band, n - 1) + 1):
        w = -rng.uniform(0.5, 1.0, n - d)
        i = np.arange(n - d)
        rows += [i, i + d]
        cols += [i + d, i]
        vals += [w, w]
    rows, cols, vals = map(np.concatenate, (rows, cols, vals))
    o = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), cols[o].astype(np.int32), vals[o]


def product(rp, ci, v, x):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    return np.bincount(rows, weights=v * x[ci], minlength=len(rp) - 1)


def cg(rp, ci, v, b, x, its, tol):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    d = 1.0 / v[rows == ci]
    x, r = x.copy(), b - product(rp, ci, v, x)
    p, rho_old, done = np.zeros_like(b), 1.0, 0
    while done < its and np.linalg.norm(r) > tol * np.linalg.norm(b):
        z = d * r
        rho = r @ z
        p = z + rho / rho_old * p
        q = product(rp, ci, v, p)
        a = rho / (p @ q)
        x += a * p
        r -= a * q
        rho_old = rho
        done += 1
    return x, done


def solver(exe, A, its, tol):
    return (Cg.build().with_criteria(Iteration.build().with_max_iters(its),
                                     ResidualNorm.build().with_reduction_factor(tol))
            .with_preconditioner(Jacobi.build().with_max_block_size(1)).on(exe).generate(A))


# 148 SMs: 32 rows per block up to 4,736 rows; 512 threads per block, so one
# row per thread up to 75,776, two to 151,552, four to 303,104; the matrix in
# 224 KB per block (band 40: 81 * 12 bytes per row)
@pytest.mark.parametrize("n,band", [(1, 1), (2, 1), (33, 1), (1000, 4), (4736, 1), (4737, 13),
                                    (9473, 2), (18945, 1), (30000, 40), (75776, 1), (75777, 3),
                                    (151553, 1), (303104, 1), (303105, 1), (70000, 13)])
@pytest.mark.parametrize("its", [1, 2, 9, 200])
def test_one_column(n, band, its):
    exe = CudaExecutor.create(0)
    rp, ci, v = banded(n, band, n)
    rng = np.random.default_rng(its)
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    x = torch.from_numpy(x0).cuda()
    s = solver(exe, Csr.read(exe, rp, ci, v), its, 1e-12)
    s.apply(torch.from_numpy(b).cuda(), x)
    ref, done = cg(rp, ci, v, b, x0, its, 1e-12)
    assert abs(s.logger.num_iterations - done) <= (0 if its < 200 else 1)
    # strictly dominant rows: a well-conditioned recurrence, both sides within
    # a few eps of each other per iteration or within the tolerance at the end
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("n,band,k", [(50, 1, 4), (98304, 1, 4), (98303, 1, 4), (24577, 1, 16),
                                      (98305, 3, 3), (3100, 13, 16), (12289, 13, 4),
                                      (140000, 4, 8), (600000, 1, 1)])
@pytest.mark.parametrize("its", [1, 2, 300])
def test_columns_stop_apart(n, band, k, its):
    exe = CudaExecutor.create(0)
    rp, ci, v = banded(n, band, n)
    rng = np.random.default_rng(k)
    b, x0 = rng.standard_normal((n, k)), rng.standard_normal((n, k))
    if k > 1:
        b[:, 0] = product(rp, ci, v, x0[:, 0])  # starts at the solution
        near = x0[:, 1] + 1e-6 * rng.standard_normal(n)
        b[:, 1] = product(rp, ci, v, near)      # stops early
    wide = torch.full((n, k + 1), 7.0, dtype=torch.float64, device="cuda")
    x = wide[:, :k]
    x.copy_(torch.from_numpy(x0))
    s = solver(exe, Csr.read(exe, rp, ci, v), its, 1e-12)
    s.apply(torch.from_numpy(b).cuda(), x)
    got = x.cpu().numpy()
    for j in range(k):
        ref, _ = cg(rp, ci, v, b[:, j], x0[:, j], its, 1e-12)
        assert np.linalg.norm(got[:, j] - ref) <= 1e-10 * np.linalg.norm(ref), j
    assert bool((wide[:, k] == 7.0).all())


@pytest.mark.parametrize("n", [700, 75777])
def test_rows_longer_than_said(n):
    """An understated longest row must not size the resident kernel's stage."""
    exe = CudaExecutor.create(0)
    rp, ci, v = banded(n, 2, n)
    b = np.random.default_rng(3).standard_normal(n)
    A = Csr.read(exe, rp, ci, v)
    A._max_row_nnz = 1
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    s = solver(exe, A, 200, 1e-12)
    s.apply(torch.from_numpy(b).cuda(), x)
    ref, _ = cg(rp, ci, v, b, np.zeros(n), 200, 1e-12)
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1e-10 * np.linalg.norm(ref)
