"""Batched BiCGStab with the matrix staged in shared memory against the form
that reads it from global memory: the same systems at the edges of the size
buckets, stored with five entries per row (staged) and with 64 (too wide to
stage above a few hundred rows), the padding holding NaN values and columns
outside the system."""
import numpy as np
import pytest
import torch

from ginkgo_b200 import stencils
from ginkgo_b200.batch import BatchBicgstab, BatchEll
from ginkgo_b200.matrix import CudaExecutor
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513, 1000, 1023, 1024]


@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
@pytest.mark.parametrize("copies", [1, 40])
def test_staged_and_global_matrix_agree(dt, copies):
    exe = CudaExecutor.create(0)
    rng = np.random.default_rng(4)
    systems = []
    for n in SIZES * copies:
        nx, ny = stencils.most_square_grid(n)
        rp, ci, v = stencils.convection_diffusion_2d(nx, ny, 1.0, *rng.uniform(-1, 1, 2))
        # I + L: rows dominant by one, so max |A^-1 e| <= max |e|
        v = v + (ci == np.repeat(np.arange(n), np.diff(rp)))
        systems.append((rp, ci, v))
    narrow = BatchEll.from_csr(exe, systems, width=5, dtype=dt)
    wide = BatchEll.from_csr(exe, systems, width=64, dtype=dt)
    pad = wide.col_idxs == -1
    wide.values[pad] = float("nan")
    wide.col_idxs[pad] = torch.from_numpy(
        rng.choice([-1, -7, 5000], int(pad.sum())).astype(np.int32)).cuda()
    b = torch.from_numpy(rng.standard_normal(narrow.total_rows)).to(dt).cuda()
    tol = 1e-10 if dt == torch.float64 else 1e-5
    xs = []
    for A in (narrow, wide):
        x = torch.zeros_like(b)
        s = (BatchBicgstab.build().with_max_iterations(200).with_tolerance(tol)
             .with_tolerance_type("relative").with_preconditioner("jacobi").on(exe).generate(A))
        s.apply(b, x)
        assert int(s.logger.iterations.max()) < 200
        xs.append(x.cpu().numpy().astype(np.float64))
    bh, offs = b.cpu().numpy().astype(np.float64), narrow.host_row_offsets
    npdt = np.float64 if dt == torch.float64 else np.float32
    for i, (rp, ci, v) in enumerate(systems):
        o, e = offs[i], offs[i + 1]
        norm = np.linalg.norm(bh[o:e])
        # each solution is within max |A^-1 r| <= ||r|| <= tol ||b|| of the
        # exact one, plus the drift of the recursive residual: a few eps of
        # the largest iterate times the iterations
        allow = (tol + 100 * np.finfo(npdt).eps) * norm
        assert np.abs(xs[0][o:e] - xs[1][o:e]).max() <= 2 * allow, (i, e - o)
        r = bh[o:e] - orc.csr_spmv(rp, ci, v.astype(npdt).astype(np.float64), xs[0][o:e])
        assert np.linalg.norm(r) <= 10 * allow, (i, e - o)  # ||A|| <= 10
