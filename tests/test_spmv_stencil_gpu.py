"""The unrolled SpMV of 5- and 7-point stencils (uniform diagonals) at the edges of its slices (64
rows FP64, 128 rows FP32): grid sizes around them, offsets that are and are not multiples of the
vector width, rectangular row ranges, x at every alignment, entries of x that no row may touch."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from hethyppar_gb300 import Matrix, bicgstab, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

GRIDS = [(10, 10), (16, 16), (64, 33), (127, 65), (128, 64), (129, 31), (300, 301),
         (12, 12, 12), (20, 21, 22), (33, 32, 31), (64, 64, 17)]


def _rows(rp, col, val, m):
    return rp[:m + 1], col[:rp[m]], val[:rp[m]]


@pytest.mark.parametrize("dims", GRIDS, ids=["x".join(map(str, d)) for d in GRIDS])
def test_stencil_spmv(ctx, dims):
    rp, col, val = synth._stencil(dims, 20.0, (1.0, 0.5, 0.25)[:len(dims)])
    n = rp.size - 1
    rng = np.random.default_rng(n)
    val = val * rng.uniform(0.5, 1.5, val.size)
    x = rng.standard_normal(n)
    for m in (n, n - 1, n - 3, n - 63):  # whole, and row ranges whose last slice is ragged
        rpm, cm, vm = _rows(rp, col, val, m)
        A = Matrix.from_csr(ctx, rpm, cm, vm, shape=(m, n))
        ref = orc.spmv(rpm, cm, vm, x, fma=True)
        assert np.array_equal(A.spmv(x), ref)
        y0 = rng.standard_normal(m)
        for off in (0, 1):  # 16- and 8-byte aligned x
            xd = torch.zeros(n + 2, dtype=torch.float64, device="cuda")[off:off + n]
            xd.copy_(dev(x))
            y = dev(y0)
            A.spmv_dev(xd, y, alpha=1.5, beta=-2.0)
            want = np.array([np.float64(-2.0) * b for b in y0]) + 1.5 * ref
            tol = 4.5e-16 * (np.abs(2.0 * y0) + np.abs(1.5 * ref))
            assert np.all(np.abs(y.cpu().numpy() - want) <= tol)
            A.spmv_dev(xd, y)
            assert np.array_equal(y.cpu().numpy(), ref)
        # FP32: sequential sums of at most 7 products: 8 roundings of the largest partial sum
        x32, v32 = x.astype(np.float32), vm.astype(np.float32)
        exact = orc.spmv(rpm, cm, v32.astype(np.float64), x32.astype(np.float64))
        bound = 8 * 2.0 ** -24 * orc.spmv(rpm, cm, np.abs(v32).astype(np.float64), np.abs(x32).astype(np.float64))
        first = None
        for off in range(4):
            xd = torch.zeros(n + 4, dtype=torch.float32, device="cuda")[off:off + n]
            xd.copy_(dev(x32, torch.float32))
            y = torch.full((m,), float("nan"), dtype=torch.float32, device="cuda")
            A.spmv_f32_dev(xd, y)
            got = y.cpu().numpy()
            assert np.all(np.abs(got - exact) <= bound)
            first = got if first is None else first
            assert np.array_equal(got, first)
        A.close()


def test_absent_entries_are_not_touched(ctx):
    """A row without an entry on some diagonal ignores x there, whatever it holds."""
    rp, col, val = synth._stencil((96, 40), 20.0, (1.0, 0.5))
    n = rp.size - 1
    x = np.random.default_rng(0).standard_normal(n)
    # NaN at a grid corner: rows 0, 1 and 96 store it; the end of the last row's neighbour does not
    x[0] = np.nan
    A = Matrix.from_csr(ctx, rp, col, val)
    y = A.spmv(x)
    bad = np.array([0 in col[a:b] for a, b in zip(rp[:-1], rp[1:])])
    assert np.array_equal(np.isnan(y), bad)
    x[0], x[95] = 1.0, np.inf  # the last point of the first grid row: row 96 is its diagonal neighbour
    y, ref = A.spmv(x), orc.spmv(rp, col, val, x, fma=True)
    assert np.array_equal(y, ref)
    A.close()


def test_values_refresh_and_dropped_csr(ctx):
    s = synth.convdiff3d(24, 20.0, seed=3)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    A.spmv(s.x_target)
    v2 = s.val * np.random.default_rng(1).uniform(0.9, 1.1, s.val.size)
    A.set_values(v2)
    assert np.array_equal(A.spmv(s.x_target), orc.spmv(s.rowptr, s.col, v2, s.x_target, fma=True))
    A.set_values(s.val)
    x, r = bicgstab(ctx, A, s.b, rtol=1e-10)
    A.drop_csr(keep_fp32=True)
    x2, r2 = bicgstab(ctx, A, s.b, rtol=1e-10)
    assert np.array_equal(x, x2) and r.iters == r2.iters
    A.close()


@pytest.mark.parametrize("offsets", [(0, 1, 2, 3, 4), (-3, -2, -1, 0, 1), (-64, -2, 0, 2, 64), (-9, -1, 0, 1, 2),
                                     (-65, -1, 0, 1, 66), (-100, -7, -1, 0, 1, 7, 100), (-96, -8, -2, 0, 3, 8, 96),
                                     (-3, -2, -1, 0, 1, 2, 3), (-5, -4, -3, -1, 0, 1, 2)])
def test_middle_diagonals(ctx, offsets):
    """Diagonals beside the main one share its words of x; other sets of 5 and 7 do not."""
    n = 128 * 70 + 37
    rng = np.random.default_rng(n)
    cols = np.arange(n)[:, None] + np.array(offsets)
    keep = (cols >= 0) & (cols < n) & (rng.random(cols.shape) > 0.03)
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    col = cols[keep].astype(np.int32)
    val, x = rng.standard_normal(col.size), rng.standard_normal(n)
    A = Matrix.from_csr(ctx, rp, col, val, shape=(n, n))
    assert np.array_equal(A.spmv(x), orc.spmv(rp, col, val, x, fma=True))
    x32, v32 = x.astype(np.float32), val.astype(np.float32)
    exact = orc.spmv(rp, col, v32.astype(np.float64), x32.astype(np.float64))
    bound = 8 * 2.0 ** -24 * orc.spmv(rp, col, np.abs(v32).astype(np.float64), np.abs(x32).astype(np.float64))
    first = None
    for off in range(4):
        xd = torch.zeros(n + 4, dtype=torch.float32, device="cuda")[off:off + n]
        xd.copy_(dev(x32, torch.float32))
        y = torch.full((n,), float("nan"), dtype=torch.float32, device="cuda")
        A.spmv_f32_dev(xd, y)
        got = y.cpu().numpy()
        assert np.all(np.abs(got - exact) <= bound)
        first = got if first is None else first
        assert np.array_equal(got, first)
    A.close()


@pytest.mark.parametrize("dims", [(550, 40, 40), (600, 40, 40), (985, 40, 40)])
def test_loop_kernel_by_size(ctx, dims):
    """Systems on both sides of the sizes whose loop products take the general kernel: the first iterations
    of both schedules as the reference's loop has them."""
    rp, col, val = synth._stencil(dims, 20.0, (1.0, 0.5, 0.25))
    n = rp.size - 1
    b = np.random.default_rng(n).standard_normal(n)
    ref = orc.bicgstab_fixed(rp, col, val, b, np.zeros(n), 3)[0]
    A = Matrix.from_csr(ctx, rp, col, val)
    for loop in ("merged", "classic"):
        x, r = bicgstab(ctx, A, b, rtol=1e-12, maxit=3, loop=loop)
        assert r.iters == 3 and np.max(np.abs(x - ref)) <= 1e-10 * max(1.0, np.max(np.abs(ref)))
    A.close()


@pytest.mark.parametrize("dims", [(580, 50, 50), (590, 50, 50), (1040, 50, 50), (1055, 50, 50)])
def test_product_kernel_by_size(ctx, dims):
    """Plain products on both sides of the sizes that take the general kernel: row sums bit for bit."""
    rp, col, val = synth._stencil(dims, 20.0, (1.0, 0.5, 0.25))
    n = rp.size - 1
    rng = np.random.default_rng(n)
    x, y0 = rng.standard_normal(n), rng.standard_normal(n)
    A = Matrix.from_csr(ctx, rp, col, val)
    want = orc.spmv(rp, col, val, x, fma=True)
    xd, y = dev(x), torch.empty(n, dtype=torch.float64, device="cuda")
    A.spmv_dev(xd, y)
    assert np.array_equal(y.cpu().numpy(), want)
    y = dev(y0)
    A.spmv_dev(xd, y, 0.5, 1.0)  # exact up to the one rounding of the sum
    assert np.array_equal(y.cpu().numpy(), 0.5 * want + y0)
    A.close()
