"""Batched BiCGStab on the largest systems that it accepts (1,025 to 2,048
rows): staged in shared memory, with the matrix in global memory, uniform, and
through the tuner."""
import numpy as np
import pytest
import torch

from ginkgo_b200 import stencils
from ginkgo_b200.batch import BatchBicgstab, BatchEll
from ginkgo_b200.matrix import CudaExecutor
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [1024, 1025, 1500, 2047, 2048, 3]


def system(n, rng):
    nx, ny = stencils.most_square_grid(n)
    rp, ci, v = stencils.convection_diffusion_2d(nx, ny, 1.0, *rng.uniform(-1, 1, 2))
    # I + L: rows dominant by one, so ||A^-1 r||_inf <= ||r||_inf
    return rp, ci, v + (ci == np.repeat(np.arange(n), np.diff(rp)))


def solver(exe, A, tol):
    return (BatchBicgstab.build().with_max_iterations(200).with_tolerance(tol)
            .with_tolerance_type("relative").with_preconditioner("jacobi").on(exe).generate(A))


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("form", ["width5", "width24", "tuned", "uniform"])
def test_large_systems(form, dt):
    exe = CudaExecutor.create(0)
    rng = np.random.default_rng(3)
    npdt = np.float64 if dt == torch.float64 else np.float32
    systems = [system(2048 if form == "uniform" else n, rng) for n in SIZES]
    A = BatchEll.from_csr(exe, systems, width=24 if form == "width24" else 5, dtype=dt)
    if form == "uniform":
        A = BatchEll.uniform(exe, len(systems), 2048, 5, A.col_idxs[:2048 * 5], A.values)
    b = torch.from_numpy(rng.standard_normal(A.total_rows)).to(dt).cuda()
    tol = 1e-10 if dt == torch.float64 else 1e-5
    s = solver(exe, A, tol)
    x = torch.zeros_like(b)
    if form == "tuned":
        s.tune(b, x)
        x.zero_()
    s.apply(b, x)
    assert int(s.logger.iterations.max()) < 200
    bh, xh = (t.cpu().numpy().astype(np.float64) for t in (b, x))
    for i, (rp, ci, v) in enumerate(systems):
        o, e = A.host_row_offsets[i], A.host_row_offsets[i + 1]
        r = bh[o:e] - orc.csr_spmv(rp, ci, v.astype(npdt).astype(np.float64), xh[o:e])
        # the tolerance, plus the drift of the recursive residual: a few eps
        # of ||A|| (at most 10) times the iterates, over at most 100 iterations
        allow = (tol + 100 * 10 * np.finfo(npdt).eps) * np.linalg.norm(bh[o:e])
        assert np.linalg.norm(r) <= allow, (i, e - o)
