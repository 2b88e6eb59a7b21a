"""GMRES and IR on matrices that take the slice-offset copy (32 rows share one
list of column offsets) and on matrices that the copy refuses: widths on both
sides of its batches of 5, 7 and 9 slots and of a warp's 32 offsets, whole and
partial last slices, rows stored in another order, and the row count up to
which FP32 uses it.  Every case states which copy it is for; that is checked
here against the padding rule and a restatement of the fill."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor
from ginkgo_b200.solver import Gmres, Ir, Iteration, Jacobi, ResidualNorm

pytestmark = pytest.mark.gpu


def band(n, offs, order=None, edge=0):
    """Rows of the entries at `offs` that exist, in `order` (a permutation of
    the offsets); the first `edge` rows and the last slice are diagonal."""
    offs = np.asarray(offs)[slice(None) if order is None else order]
    cols = np.arange(n)[:, None] + offs[None, :]
    ok = (cols >= 0) & (cols < n)
    if edge:
        last = (n - 1) // 32 * 32
        ok[:edge] = ok[last:] = offs[None, :] == 0
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))])
    return rp, cols[ok]


def values(rp, ci):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    rng = np.random.default_rng(len(ci))
    width = int(np.diff(rp).max())
    return np.where(ci == rows, width + rng.uniform(0, 1, len(ci)),
                    rng.uniform(-1, 1, len(ci)))


def copied(n, rp):
    """Whether the padded column-major copy is made at all."""
    nnz = int(rp[-1])
    return int(np.diff(rp).max()) * (-(-n // 64) * 64) <= nnz + nnz // 4


def slots(n, rp, ci):
    """The most offsets that a slice of the fill needs."""
    most = 0
    for s in range(0, n, 32):
        seqs = [[int(c) - r for c in ci[rp[r]:rp[r + 1]]] for r in range(s, min(s + 32, n))]
        at, count = [0] * len(seqs), 0
        while any(a < len(q) for a, q in zip(at, seqs)):
            m = min(q[a] for a, q in zip(at, seqs) if a < len(q))
            at = [a + (a < len(q) and q[a] == m) for a, q in zip(at, seqs)]
            count += 1
        most = max(most, count)
    return most


def solve_and_check(n, rp, ci, storage):
    v = values(rp, ci)
    exe = CudaExecutor.create(0)
    b = np.random.default_rng(1).standard_normal(n)
    jacobi = Jacobi.build().with_max_block_size(1)
    if storage == "f32":
        f = Ir.build().with_solver(Gmres.build().with_krylov_dim(30).with_storage_precision("f32")
                                   .with_preconditioner(jacobi))
    else:
        f = Gmres.build().with_krylov_dim(30).with_preconditioner(jacobi)
    s = f.with_criteria(Iteration.build().with_max_iters(2000),
                        ResidualNorm.build().with_reduction_factor(1e-12)).on(exe).generate(
        Csr.read(exe, rp.astype(np.int32), ci.astype(np.int32), v))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    s.apply(torch.from_numpy(b).cuda(), x)
    assert s.logger.has_converged
    rows = np.repeat(np.arange(n), np.diff(rp))
    r = b - np.bincount(rows, weights=v * x.cpu().numpy()[ci], minlength=n)
    # the loop stops on the explicit FP64 residual; forming it once more
    # rounds within a few eps of ||A|| ||x||, far below 1e-12 ||b|| here
    assert np.linalg.norm(r) <= 2e-12 * np.linalg.norm(b)


BANDS = {1: [0], 4: [-2, 0, 1, 2], 5: [-3, -1, 0, 1, 3], 6: [-3, -1, 0, 1, 2, 3],
         7: list(range(-3, 4)), 8: list(range(-4, 4)), 9: list(range(-4, 5)),
         10: list(range(-5, 5)), 27: list(range(-13, 14)), 33: list(range(-16, 17)),
         41: list(range(-20, 21))}


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("width", sorted(BANDS))
@pytest.mark.parametrize("n", [62, 64, 127, 128, 371, 384])
def test_bands(n, width, storage):
    rp, ci = band(n, BANDS[width])
    if n < 100 and width > 10:
        pytest.skip("edge rows leave too much padding")
    assert copied(n, rp) and slots(n, rp, ci) <= width
    solve_and_check(n, rp, ci, storage)


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("n", [620, 640])
@pytest.mark.parametrize("order", [[4, 3, 2, 1, 0], [2, 0, 4, 1, 3]])
def test_another_order(n, order, storage):
    rp, ci = band(n, BANDS[5], order, edge=32)
    assert copied(n, rp) and slots(n, rp, ci) == 5
    solve_and_check(n, rp, ci, storage)


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("kind", ["each row its order", "random columns"])
def test_refused(kind, storage):
    n, rng = 640, np.random.default_rng(2)
    if kind == "random columns":
        ci = np.concatenate([np.sort(np.concatenate(
            [[i], rng.choice(np.delete(np.arange(n), i), 4, replace=False)])) for i in range(n)])
        rp = np.arange(n + 1) * 5
    else:
        rp, ci = band(n, BANDS[5])
        ci = np.concatenate([rng.permutation(ci[rp[r]:rp[r + 1]]) for r in range(n)])
    assert copied(n, rp) and slots(n, rp, ci) > 5
    solve_and_check(n, rp, ci, storage)


@pytest.mark.parametrize("n", [1 << 19, (1 << 19) + 1])
def test_largest_fp32_copy(n):
    rp, ci = band(n, BANDS[5])
    assert copied(n, rp)
    solve_and_check(n, rp, ci, "f32")
