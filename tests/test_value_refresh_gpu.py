"""New values reach every layout: rows of one length up to the slice limit, ragged and empty rows, rows
that long rows or the sorting take out of order; FP64, FP32 before and after its first use, and the
transpose."""
import numpy as np
import pytest

from hethyppar_gb300 import Matrix, bicgstab_backward
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _spmv32(A, x):
    import torch

    y = torch.empty(A.shape[0], dtype=torch.float32, device="cuda")
    A.spmv_f32_dev(torch.as_tensor(x, dtype=torch.float32, device="cuda"), y)
    return y.cpu().numpy()


def _lens(kind, m, rng):
    if kind == "ragged":
        return rng.integers(20, 25, m) * (rng.random(m) > 0.02)
    if kind == "long":
        lens = np.full(m, 20)
        lens[[m // 3, m // 2]] = 6000
        return lens
    if kind == "sorted":
        return rng.choice([1, 4, 60], m)
    return np.full(m, kind)


KINDS = [1, 2, 15, 16, 29, 30, 31, 32, 33, 48, 64, 700, "ragged", "long", "sorted"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("m", [1, 31, 33, 129, 4097])
def test_values(ctx, kind, m):
    if kind == 700 and m > 129:
        m = 200
    rng = np.random.default_rng(m)
    n = 7000
    lens = _lens(kind, m, rng)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    start = rng.integers(0, n - 6000, m)
    col = (np.repeat(start - rp[:-1], lens) + np.arange(rp[-1])).astype(np.int32)
    v1, v2 = rng.standard_normal(rp[-1]), rng.standard_normal(rp[-1])
    x = rng.standard_normal(n)
    A = Matrix.from_csr(ctx, rp, col, v1, shape=(m, n))
    B = Matrix.from_csr(ctx, rp, col, v2, shape=(m, n))
    A.spmv(x)
    A.set_values(v2)  # the FP64 layout alone exists
    y = A.spmv(x)
    assert np.array_equal(y, B.spmv(x))
    mag = orc.spmv(rp, col, np.abs(v2), np.abs(x))
    # sums of k terms in another order: each is within k rounding errors of the magnitudes' sum
    assert np.all(np.abs(y - orc.spmv(rp, col, v2, x)) <= 2 * (lens + 4) * 2.0**-53 * mag)
    y32 = _spmv32(A, x)
    assert np.array_equal(y32, _spmv32(B, x))
    A.set_values(v1)
    A.set_values(v2)  # both layouts exist
    assert np.array_equal(y32, _spmv32(A, x))
    assert np.array_equal(y, A.spmv(x))
    A.close()
    B.close()


@pytest.mark.parametrize("m", [100, 5000])
def test_transpose(ctx, m):
    rng = np.random.default_rng(m)
    k = 16
    col = np.sort((np.arange(m)[:, None] + np.arange(-(k // 2), k - k // 2)) % m, axis=1).astype(np.int32)
    rp = np.arange(0, m * k + 1, k, dtype=np.int32)
    diag = col.ravel() == np.repeat(np.arange(m), k)

    def values():
        v = rng.uniform(-1.0, 1.0, m * k)
        v[diag] = 12.0
        return v

    v1, v2 = values(), values()
    x, g = rng.standard_normal(m), rng.standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col.ravel(), v1)
    B = Matrix.from_csr(ctx, rp, col.ravel(), v2)
    for precision in ("fp64", "mixed"):
        bicgstab_backward(ctx, A, x, g, rtol=1e-10, maxit=300, precision=precision)
        A.set_values(v2)
        a = bicgstab_backward(ctx, A, x, g, rtol=1e-10, maxit=300, precision=precision)
        b = bicgstab_backward(ctx, B, x, g, rtol=1e-10, maxit=300, precision=precision)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and a[2].status == 0
        A.set_values(v1)
    A.close()
    B.close()
