"""GMRES and IR on the slice-offset copy of the matrix (bands, sizes that
leave part of a slice, unsorted rows) and on the patterns that it refuses,
against a dense solve."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Gmres, Ir, Iteration, Jacobi, ResidualNorm

pytestmark = pytest.mark.gpu


def matrix(kind, n, seed):
    rng = np.random.default_rng(seed)
    rows = np.arange(n)
    if kind == "random":
        # five entries per row, no offsets in common: wider than the copy
        cols = [np.sort(np.concatenate([[i], rng.choice(np.delete(rows, i), 4, replace=False)]))
                for i in rows]
    else:
        far = max(n // 3, 2)
        offs = [-far, -1, 0, 1, far] if kind != "wide" else list(range(-20, 21))
        cols = [np.array([i + o for o in offs if 0 <= i + o < n]) for i in rows]
        if kind == "unsorted":
            cols = [rng.permutation(c) for c in cols]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    r = np.repeat(rows, np.diff(rp))
    v = np.where(ci == r, len(cols[n // 2]) + rng.uniform(0, 1, len(ci)),
                 rng.uniform(-1, 1, len(ci)))
    return rp, ci, v


@pytest.mark.parametrize("kind", ["band", "wide", "unsorted", "random"])
@pytest.mark.parametrize("n", [31, 32, 33, 200, 401])
@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_solution(kind, n, storage):
    exe = CudaExecutor.create(0)
    rp, ci, v = matrix(kind, n, n)
    dense = np.zeros((n, n))
    np.add.at(dense, (np.repeat(np.arange(n), np.diff(rp)), ci), v)
    b = np.random.default_rng(1).standard_normal(n)
    crit = (Iteration.build().with_max_iters(2000),
            ResidualNorm.build().with_reduction_factor(1e-12))
    jacobi = Jacobi.build().with_max_block_size(1)
    if storage == "f32":
        f = Ir.build().with_solver(Gmres.build().with_krylov_dim(30).with_storage_precision("f32")
                                   .with_preconditioner(jacobi))
    else:
        f = Gmres.build().with_krylov_dim(30).with_preconditioner(jacobi)
    s = f.with_criteria(*crit).on(exe).generate(Csr.read(exe, rp, ci, v))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    s.apply(torch.from_numpy(b).cuda(), x)
    assert s.logger.has_converged
    # ||x - A^-1 b|| <= ||A^-1|| ||r||
    ref = np.linalg.solve(dense, b)
    allow = np.linalg.norm(np.linalg.inv(dense), 2) * 2e-12 * np.linalg.norm(b)
    assert np.linalg.norm(x.cpu().numpy() - ref) <= allow
