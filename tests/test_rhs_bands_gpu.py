"""Block SpMV at the row counts where the kernel changes (2^14 to 2^19 rows,
short and longer rows, one to eight 16-byte column slices): rows per warp, one
or two rows per lane slot, on even and odd strides, against FP64 sums."""
import pytest
import torch

from ginkgo_b200.matrix import Csr, CudaExecutor, Ell

pytestmark = pytest.mark.gpu


def banded(n, length, dt):
    """Rows of up to `length` entries at fixed offsets, the first and last
    rows shorter; every seventh row loses its first entry."""
    g = torch.Generator("cuda").manual_seed(n + length)
    offs = torch.arange(length, device="cuda") * 3 - (3 * length) // 2
    rows = torch.arange(n, device="cuda")
    cols = rows[:, None] + offs[None, :]
    ok = (cols >= 0) & (cols < n)
    ok[::7, 0] = False
    v = torch.randn(n, length, device="cuda", dtype=dt, generator=g)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(ok.sum(1), 0, out=rp[1:])
    return rp.int(), cols, ok, v


def shifted(t, by):
    """The same values on storage that starts `by` elements off alignment."""
    s = torch.empty(t.numel() + by, dtype=t.dtype, device="cuda")[by:]
    return s.copy_(t.reshape(-1))


K14, K15, K16, K17 = 1 << 14, 1 << 15, 1 << 16, 1 << 17


@pytest.mark.parametrize("dt,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("n,length", [(K14 - 1, 5), (K14, 8), (K14, 9), (K15 - 1, 12), (K15, 9),
                                      (K15 + 1, 7), (K16 - 1, 9), (K16, 3), (K16 + 1, 20),
                                      (K17 - 1, 8), (K17 - 1, 9), (K17, 8), (K17, 11),
                                      (2 * K17 - 1, 5), (2 * K17, 5), (4 * K17 - 1, 3),
                                      (4 * K17, 3), (20001, 70)])
def test_bands(n, length, dt, eps):
    exe = CudaExecutor.create(0)
    rp, cols, ok, v = banded(n, length, dt)
    A = Csr(exe, (n, n), rp, cols[ok].int(), v[ok])
    ops = {"csr": A, "sellp": A.convert_to_sellp(32), "sellp_7": A.convert_to_sellp(7, 2)}
    for name, stride in (("ell", n + n % 2), ("ell_odd", n + 1 - n % 2)):
        ops[name] = A.convert_to_ell(stride=stride)
    E = ops["ell"]
    ops["ell_off"] = Ell(exe, E.shape, E.width, E.stride, shifted(E.col_idxs, 1),
                         shifted(E.values, 1))
    for k in (4, 8, 16):
        x = torch.randn(n, k, dtype=dt, device="cuda",
                        generator=torch.Generator("cuda").manual_seed(k))
        ref = torch.zeros(n, k, dtype=torch.float64, device="cuda")
        mag = torch.zeros_like(ref)
        for d in range(length):
            term = torch.where(ok[:, d], v[:, d].double(), 0.0)[:, None] * \
                x[cols[:, d].clamp(0, n - 1)].double()
            ref += term
            mag += term.abs()
        for name, op in ops.items():
            y = torch.full((n, k), float("nan"), dtype=dt, device="cuda")
            op.apply(x, y)
            # `length` products, each rounded at most length + 1 times
            assert bool(((y.double() - ref).abs() <= (length + 1) * eps * mag).all()), (name, k)
            y.copy_(x)
            op.apply(-1.0, x, 2.0, y)
            allow = (length + 4) * eps * (mag + 2 * x.double().abs())
            assert bool(((y.double() - (2 * x.double() - ref)).abs() <= allow).all()), (name, k)
