"""The bounded waits of the one-kernel CG loop: a solve whose blocks may not
wait at all ends with an error status, leaves x as it was and the context
usable; with the default limit given by the caller it is the plain solve."""
import ctypes as C

import numpy as np
import pytest
import torch

from ginkgo_b200._lib import GinkgoError, call, lib

pytestmark = pytest.mark.gpu


def system(n, dtype):
    """Tridiagonal (-1, 4, -1)."""
    rows = np.arange(n)
    cols = np.stack([rows - 1, rows, rows + 1], 1)
    ok = (cols >= 0) & (cols < n)
    v = np.broadcast_to([-1.0, 4.0, -1.0], cols.shape)[ok]
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))])
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a)).to(d).cuda()  # noqa: E731
    return t(rp, torch.int32), t(cols[ok], torch.int32), t(v, dtype)


@pytest.mark.parametrize("dt,sfx", [(torch.float64, "f64"), (torch.float32, "f32")])
@pytest.mark.parametrize("n", [20, 33, 4737, 75777])  # 1, 2 and all blocks; rows per thread
def test_wait_limit(dt, sfx, n):
    rp, ci, v = system(n, dt)
    b = torch.randn(n, dtype=dt, device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    ws = torch.empty(lib().b2s_cg_workspace_bytes(n, 1, b.element_size()), dtype=torch.uint8,
                     device="cuda")
    its, res, st = np.zeros(1, np.int64), np.zeros(1), np.zeros(1, np.uint8)
    out = [a.ctypes.data_as(C.c_void_p) for a in (its, res, st)]
    stream = torch.cuda.current_stream().cuda_stream

    def solve(x, *limit):
        call(f"b2s_cg_solve{'_waiting' if limit else ''}_{sfx}", n, rp.data_ptr(), ci.data_ptr(),
             v.data_ptr(), 3, None, b.data_ptr(), 1, x.data_ptr(), 1, 1, 50, 1e-6, 0, 8,
             ws.data_ptr(), ws.numel(), *out, stream, *limit)
        return int(its[0])

    x = torch.full((n,), 0.25, dtype=dt, device="cuda")
    with pytest.raises(GinkgoError, match="did not meet"):
        solve(x, 0)
    assert bool((x == 0.25).all())
    with pytest.raises(GinkgoError, match="max_polls"):
        solve(x, -1)
    y = x.clone()
    assert solve(x) == solve(y, 1 << 21) < 50
    assert torch.equal(x, y)  # fixed order of every sum
