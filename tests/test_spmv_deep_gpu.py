"""SpMV (FP64 and FP32) of length-sorted matrices: rows at the edges of the groups of steps (4 and 8), of the
slice limit (256 entries) and of the chunks beyond it, on short matrices (the deep kernel) and on a
long one (the ordinary one), with all epilogues through a solve."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from hethyppar_gb300 import Matrix, bicgstab
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 15, 16, 17, 23, 31, 33, 63, 65, 127, 250, 255, 256, 257, 300]


def _matrix(m, n, pool, seed, far):
    rng = np.random.default_rng(seed)
    lens = rng.choice(pool, size=m)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    if far:
        col = rng.integers(0, n, size=int(rp[-1]))
    else:  # within 16-bit distance of the row
        col = np.clip(np.repeat(np.arange(m), lens) + rng.integers(-300, 301, size=int(rp[-1])), 0, n - 1)
    return rp, col.astype(np.int32), rng.standard_normal(int(rp[-1]))


@pytest.mark.parametrize("m,pool", [(40, EDGES), (1000, EDGES), (30_000, EDGES), (30_000, EDGES[:8]), (400_000, EDGES[:20])])
@pytest.mark.parametrize("far", [False, True])
def test_rows_at_the_edges(ctx, m, pool, far):
    n = max(m, 500)
    rp, col, val = _matrix(m, n, pool, m + far, far)
    x = np.random.default_rng(1).standard_normal(n)
    A = Matrix.from_csr(ctx, rp, col, val, shape=(m, n))
    y, ref = A.spmv(x), orc.spmv(rp, col, val, x, fma=True)
    short = np.diff(rp) <= 256
    assert np.array_equal(y[short], ref[short])
    bound = 2.0 * np.diff(rp) * 2.3e-16 * orc.spmv(rp, col, np.abs(val), np.abs(x))
    assert np.all(np.abs(y - ref) <= bound)
    # FP32: at most one rounding per entry of a partial sum of magnitude sum |a x|, one for the store
    x32, v32 = x.astype(np.float32), val.astype(np.float32)
    exact = orc.spmv(rp, col, v32.astype(np.float64), x32.astype(np.float64))
    bound = (np.diff(rp) + 1) * 2.0 ** -24 * 1.01 * orc.spmv(rp, col, np.abs(v32).astype(np.float64),
                                                             np.abs(x32).astype(np.float64))
    y32 = torch.empty(m, dtype=torch.float32, device="cuda")
    A.spmv_f32_dev(dev(x32, torch.float32), y32)
    assert np.all(np.abs(y32.cpu().numpy() - exact) <= bound)
    A.close()


@pytest.mark.parametrize("loop", ["merged", "classic"])
def test_solve_on_edge_rows(ctx, loop):
    m = 3000
    rp, col, val = _matrix(m, m, EDGES, 9, True)
    rows = np.repeat(np.arange(m), np.diff(rp))
    off = np.bincount(rows, weights=np.abs(val), minlength=m)
    rp2 = (rp + np.arange(m + 1)).astype(np.int32)
    at = rp2[1:] - 1  # the diagonal as each row's last entry
    c2, v2 = np.empty(rp2[-1], np.int32), np.empty(rp2[-1])
    body = np.ones(rp2[-1], bool)
    body[at] = False
    c2[body], v2[body], c2[at], v2[at] = col, val, np.arange(m), 1.5 * off + 1.0
    b = np.random.default_rng(2).standard_normal(m)
    A = Matrix.from_csr(ctx, rp2, c2, v2)
    x, r = bicgstab(ctx, A, b, rtol=1e-12, loop=loop)
    assert r.status == 0
    res = b - orc.spmv(rp2, c2, v2, x)
    assert np.sqrt(orc.dot(res, res) / orc.dot(b, b)) <= 1.0000001e-12
    x, r = bicgstab(ctx, A, b, rtol=1e-12, loop=loop, precision="mixed")
    assert r.status == 0
    res = b - orc.spmv(rp2, c2, v2, x)
    assert np.sqrt(orc.dot(res, res) / orc.dot(b, b)) <= 1.0000001e-12
    A.close()
