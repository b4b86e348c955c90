"""The mixed form of small systems in one kernel: every grid and cluster size, both schedules, all ways to end,
restarts and the hand-over to FP64, new values, a dropped CSR, and the same bits however it is launched."""
import numpy as np
import pytest

from hethyppar_gb300 import Matrix, bicgstab, bicgstab_backward, synth
from oracle import oracle as orc
from test_small_solve_gpu import SIZES, _dominant, _rel

pytestmark = pytest.mark.gpu
LOOPS = pytest.mark.parametrize("loop", ["merged", "classic"])


def _mixed(ctx, A, b, x0=None, rtol=1e-11, **kw):
    return bicgstab(ctx, A, b, x0, rtol=rtol, precision="mixed", **kw)


@pytest.mark.parametrize("m,width", SIZES + [(16_384, 4), (16_385, 4)])
@LOOPS
def test_sizes(ctx, m, width, loop):
    rp, col, val = _dominant(m, width, m + width)
    rng = np.random.default_rng(m)
    b, x0 = rng.standard_normal(m), rng.standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    _, r64 = bicgstab(ctx, A, b, x0, rtol=1e-11, loop=loop)
    x, r = _mixed(ctx, A, b, x0, loop=loop)
    # the mixed form's iteration bar
    assert r.status == 0 and r.iters <= 1.35 * r64.iters + 5 and r.outer_iters >= 1
    assert m <= 2 or not r.fp64_fallback  # one or two unknowns: s vanishes in FP32 before an update is due
    assert _rel(rp, col, val, b, x) <= 1.0000001e-11 and r.rel_res_true <= 1e-11
    x2, r2 = _mixed(ctx, A, b, x0, loop=loop)
    assert np.array_equal(x, x2) and r.iters == r2.iters
    xz, rz = _mixed(ctx, A, b, loop=loop)
    assert rz.status == 0 and _rel(rp, col, val, b, xz) <= 1.0000001e-11
    A.close()


@pytest.mark.parametrize("n", [24, 100])
@LOOPS
def test_ways_to_end(ctx, monkeypatch, n, loop):
    s = synth.convdiff2d(n, 30.0, seed=1)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    n0 = ctx.kernel_launches
    full, rf = _mixed(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert rf.status == 0 and rf.outer_iters >= 2 and ctx.kernel_launches - n0 <= 4
    monkeypatch.setenv("HHP_SOLVE_GRAPH", "0")
    xd, rd = _mixed(ctx, A, s.b, rtol=1e-10, loop=loop)
    monkeypatch.delenv("HHP_SOLVE_GRAPH")
    assert np.array_equal(full, xd) and (rd.iters, rd.outer_iters) == (rf.iters, rf.outer_iters)
    # the iteration cap: x is folded and its residual the true one
    for k in (0, 1, 2, 7):
        x, r = _mixed(ctx, A, s.b, rtol=1e-10, maxit=k, loop=loop)
        assert r.status == 6 and r.iters == k
        ref = orc.bicgstab_fixed(s.rowptr, s.col, s.val, s.b, np.zeros(s.n), k)[0] if k else np.zeros(s.n)
        # FP32 recurrences: 7 steps of some 20 roundings of 2^-24, amplified by the steps' growth of the residual
        assert np.max(np.abs(x - ref)) <= 1e-3 * max(1.0, np.max(np.abs(ref)))
        assert abs(_rel(s.rowptr, s.col, s.val, s.b, x) - r.rel_res_true) <= 1e-9
    x, r = _mixed(ctx, A, s.b, full, rtol=1e-9, loop=loop)
    assert r.status == 0 and r.iters == 0 and np.array_equal(x, full)
    b = s.b.copy()
    b[5] = np.nan
    assert _mixed(ctx, A, b, rtol=1e-10, loop=loop, raise_on_error=False)[1].status == 5
    Z = Matrix.from_csr(ctx, s.rowptr, s.col, np.zeros_like(s.val))
    assert _mixed(ctx, Z, s.b, rtol=1e-10, loop=loop, raise_on_error=False)[1].status == 5
    Z.close()
    # below what rounding allows: the FP32 passes stagnate, FP64 takes over, and no success is reported
    x, r = _mixed(ctx, A, s.b, rtol=1e-17, maxit=2000, loop=loop)
    assert r.status in (5, 6) and r.fp64_fallback and _rel(s.rowptr, s.col, s.val, s.b, x) <= 1e-12
    # new values and a dropped CSR
    A.set_values(2.0 * s.val)
    x, r = _mixed(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert r.status == 0 and np.array_equal(2.0 * x, full) and r.iters == rf.iters
    A.drop_csr(keep_fp32=True)
    xk, rk = _mixed(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert np.array_equal(xk, x) and rk.iters == r.iters
    A.close()


@pytest.mark.parametrize("m", [500, 16_000])
@LOOPS
def test_infinite_entry(ctx, m, loop):
    rp, col, val = _dominant(m, 4, m)
    val[rp[m // 2]] = np.inf
    b = np.random.default_rng(m).standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    for x0 in (np.zeros(m), np.ones(m)):
        x, r = _mixed(ctx, A, b, x0, rtol=1e-10, loop=loop, raise_on_error=False)
        assert r.status == 5 and r.iters == 0 and np.array_equal(x, x0)
    A.close()


@pytest.mark.parametrize("m", [50, 3000, 16_000])
@LOOPS
def test_length_sorted_rows_and_adjoint(ctx, m, loop):
    rng = np.random.default_rng(m)
    lens = np.minimum(rng.choice([1, 2, 3, 9, 17, 31], size=m), m)
    cols = []
    for i, k in enumerate(lens):
        c = rng.choice(m, size=k - 1, replace=False)
        cols.append(np.concatenate([np.sort(c[c != i]), [i]]))
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = rng.uniform(-1.0, 0.0, col.size)
    rows = np.repeat(np.arange(m), np.diff(rp))
    off = np.bincount(rows[col != rows], weights=np.abs(val[col != rows]), minlength=m)
    val[col == rows] = 1.3 * off + 0.5
    b, g = rng.standard_normal(m), rng.standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    x, r = _mixed(ctx, A, b, loop=loop)
    assert r.status == 0 and _rel(rp, col, val, b, x) <= 1.0000001e-11
    dldb, dlda, ra = bicgstab_backward(ctx, A, x, g, rtol=1e-11, precision="mixed", loop=loop)
    tr, tc, tv = orc.csr_to_csc(rp, col, val, m)
    assert ra.status == 0 and _rel(tr, tc, tv, g, dldb) <= 1.0000001e-11
    assert np.array_equal(dlda, -(dldb[rows] * x[col]))
    A.close()
