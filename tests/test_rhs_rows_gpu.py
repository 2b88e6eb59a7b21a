"""Block SpMV at the edges of the kernel choice for four or more columns:
rows per warp change with the row count (16,384) and the longest row (8 and
64 entries); ragged rows, empty rows and sizes that leave part of a warp."""
import numpy as np
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor

pytestmark = pytest.mark.gpu


def ragged(n, longest, seed):
    """Row lengths 0..longest (the first row the longest), sorted columns."""
    rng = np.random.default_rng(seed)
    m = max(n, longest)
    lens = rng.integers(0, longest + 1, n)
    lens[0] = longest
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(m, k, replace=False)) if m < 500 else
                         (rng.integers(0, m) + np.sort(rng.choice(500, k, replace=False))) % m
                         for k in lens] + [np.zeros(0, np.int64)]).astype(np.int32)
    return m, rp, ci, rng.standard_normal(len(ci))


@pytest.mark.parametrize("dt,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("n,longest", [(1, 5), (3, 8), (31, 9), (129, 64), (1000, 65), (16383, 8),
                                       (16385, 9), (16384, 7), (40001, 8)])
def test_block_products(n, longest, dt, eps):
    exe = CudaExecutor.create(0)
    m, rp, ci, v = ragged(n, longest, n + longest)
    A = Csr.read(exe, rp, ci, v, shape=(n, m), dtype=dt)
    v = A.values.double().cpu().numpy()
    rows = np.repeat(np.arange(n), np.diff(rp))
    ops = {"csr": A, "ell": A.convert_to_ell(), "ell_odd": A.convert_to_ell(stride=n + 1),
           "sellp": A.convert_to_sellp(32), "sellp_7": A.convert_to_sellp(7, 2)}
    for k in (4, 8, 16, 28):
        x = np.random.default_rng(k).standard_normal((m, k))
        xd = torch.from_numpy(x).to(dt).cuda()
        x = xd.double().cpu().numpy()
        ref, mag = np.zeros((n, k)), np.zeros((n, k))
        np.add.at(ref, rows, v[:, None] * x[ci])
        np.add.at(mag, rows, np.abs(v[:, None] * x[ci]))
        y0 = torch.from_numpy(np.random.default_rng(k + 1).standard_normal((n, k))).to(dt).cuda()
        for name, op in ops.items():
            y = torch.full((n, k), float("nan"), dtype=dt, device="cuda")
            op.apply(xd, y)
            # a sum of up to `longest` products, each term rounded at most
            # longest + 1 times
            allow = (longest + 1) * eps * mag + 1e-300
            assert np.all(np.abs(y.double().cpu().numpy() - ref) <= allow), (name, k)
            y.copy_(y0)
            op.apply(-1.0, xd, 2.0, y)
            y0h = y0.double().cpu().numpy()
            allow = (longest + 4) * eps * (mag + 2 * np.abs(y0h))
            assert np.all(np.abs(y.double().cpu().numpy() - (2 * y0h - ref)) <= allow + 1e-300), \
                (name, k)
