"""The one-kernel loop of small systems at its edges: one row, one block, every cluster size, the line
between the cluster and the grid form, the largest size and the first that keeps the graph loop, the
widest rows, rows of one entry, empty off-diagonals, published and recomputed s; both schedules, all
ways to end, restarts, history, and the same bits launched directly, repeated and after a dropped CSR."""
import math

import numpy as np
import pytest

from hethyppar_gb300 import Matrix, bicgstab, bicgstab_backward, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _rel(rp, col, val, b, x):
    r = b - orc.spmv(rp, col, val, x)
    return math.sqrt(orc.dot(r, r) / orc.dot(b, b))


def _dominant(m, width, seed):
    """m rows of up to `width` off-diagonals anywhere, a dominant diagonal first in the row."""
    rng = np.random.default_rng(seed)
    cols = [np.concatenate([[i], rng.choice(m, size=min(width, m - 1), replace=False)]) for i in range(m)]
    cols = [np.concatenate([c[:1], np.sort(c[1:][c[1:] != i])]) for i, c in enumerate(cols)]
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = rng.uniform(-1.0, 0.0, col.size)
    rows = np.repeat(np.arange(m), np.diff(rp))
    off = np.bincount(rows[col != rows], weights=np.abs(val[col != rows]), minlength=m)
    val[col == rows] = 1.2 * off + 0.5
    return rp, col, val


SIZES = [(1, 0), (2, 1), (31, 3), (32, 4), (33, 4), (64, 8), (65, 9), (128, 31), (257, 5), (1024, 12), (4095, 8),
         (6144, 4), (6145, 4), (9001, 15), (20_000, 31), (40_000, 6), (40_001, 6)]


@pytest.mark.parametrize("m,width", SIZES)
@pytest.mark.parametrize("loop", ["merged", "classic"])
def test_sizes(ctx, m, width, loop):
    rp, col, val = _dominant(m, width, m + width)
    rng = np.random.default_rng(m)
    b, x0 = rng.standard_normal(m), rng.standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    k_ref, _, _ = orc.iters_to_tol(rp, col, val, b, x0, 1e-11, 300)
    x, r = bicgstab(ctx, A, b, x0, rtol=1e-11, loop=loop, record_history=True)
    assert r.status == 0 and _rel(rp, col, val, b, x) <= 1.0000001e-11
    if k_ref >= 0:  # the reference's loop has no half step: on one row it divides 0 by 0
        assert abs(r.iters - k_ref) <= max(1, math.ceil(0.05 * k_ref))
    assert len(r.history) == r.iters and (r.iters == 0 or r.half_step or r.history[-1] <= 1.0000001e-11)
    x2, r2 = bicgstab(ctx, A, b, x0, rtol=1e-11, loop=loop)
    assert np.array_equal(x, x2) and r.iters == r2.iters
    xz, rz = bicgstab(ctx, A, b, rtol=1e-11, loop=loop)
    assert rz.status == 0 and _rel(rp, col, val, b, xz) <= 1.0000001e-11
    A.close()


@pytest.mark.parametrize("m", [50, 3000, 20_000])
@pytest.mark.parametrize("loop", ["merged", "classic"])
def test_length_sorted_rows(ctx, m, loop):
    """Row lengths from 1 to 31: the layout sorts them, a thread's row is not its position."""
    rng = np.random.default_rng(m)
    lens = np.minimum(rng.choice([1, 2, 3, 9, 17, 31], size=m), m)
    cols = []
    for i, n in enumerate(lens):
        c = rng.choice(m, size=n - 1, replace=False)
        cols.append(np.concatenate([np.sort(c[c != i]), [i]]))
    rp = np.concatenate([[0], np.cumsum([c.size for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = rng.uniform(-1.0, 0.0, col.size)
    rows = np.repeat(np.arange(m), np.diff(rp))
    off = np.bincount(rows[col != rows], weights=np.abs(val[col != rows]), minlength=m)
    val[col == rows] = 1.3 * off + 0.5
    b = rng.standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    # (no bar on the count here: on these systems it moves by 10% with the summation order)
    x, r = bicgstab(ctx, A, b, rtol=1e-11, loop=loop, maxit=300)
    assert r.status == 0 and _rel(rp, col, val, b, x) <= 1.0000001e-11
    # the transpose, whose rows are sorted differently, as the adjoint solves it
    g = rng.standard_normal(m)
    dldb, dlda, ra = bicgstab_backward(ctx, A, x, g, rtol=1e-11, maxit=300, loop=loop)
    tr, tc, tv = orc.csr_to_csc(rp, col, val, m)
    assert ra.status == 0 and _rel(tr, tc, tv, g, dldb) <= 1.0000001e-11
    rows = np.repeat(np.arange(m), np.diff(rp))
    assert np.array_equal(dlda, -(dldb[rows] * x[col]))
    A.close()


@pytest.mark.parametrize("n", [24, 100])
@pytest.mark.parametrize("loop", ["merged", "classic"])
def test_ways_to_end(ctx, monkeypatch, n, loop):
    s = synth.convdiff2d(n, 30.0, seed=1)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    full, rf = bicgstab(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert rf.status == 0
    # launched kernel by kernel: the same bits
    monkeypatch.setenv("HHP_SOLVE_GRAPH", "0")
    xd, rd = bicgstab(ctx, A, s.b, rtol=1e-10, loop=loop)
    monkeypatch.delenv("HHP_SOLVE_GRAPH")
    assert np.array_equal(full, xd) and rd.iters == rf.iters
    # the iteration cap: the first iterations of the full solve, residual as the oracle's loop has it
    for k in (0, 1, 2, 7):
        x, r = bicgstab(ctx, A, s.b, rtol=1e-10, maxit=k, loop=loop)
        assert r.status == 6 and r.iters == k
        ref = orc.bicgstab_fixed(s.rowptr, s.col, s.val, s.b, np.zeros(s.n), k)[0] if k else np.zeros(s.n)
        assert np.max(np.abs(x - ref)) <= 1e-10 * max(1.0, np.max(np.abs(ref)))
    # an exact start ends at once; a start already within the tolerance too
    x, r = bicgstab(ctx, A, s.b, full, rtol=1e-9, loop=loop)
    assert r.status == 0 and r.iters == 0 and np.array_equal(x, full)
    # breakdown: NaN in b, and (r0, v) = 0
    b = s.b.copy()
    b[5] = np.nan
    assert bicgstab(ctx, A, b, rtol=1e-10, loop=loop, raise_on_error=False)[1].status == 5
    Z = Matrix.from_csr(ctx, s.rowptr, s.col, np.zeros_like(s.val))
    assert bicgstab(ctx, Z, s.b, rtol=1e-10, loop=loop, raise_on_error=False)[1].status == 5
    Z.close()
    # a tolerance below what rounding allows: restarts, then stagnation is reported, not success
    x, r = bicgstab(ctx, A, s.b, rtol=1e-17, maxit=2000, loop=loop)
    assert r.status == 6 and r.outer_iters >= 1 and _rel(s.rowptr, s.col, s.val, s.b, x) <= 1e-12
    # new values, then a dropped CSR
    A.set_values(2.0 * s.val)
    x, r = bicgstab(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert r.status == 0 and _rel(s.rowptr, s.col, 2.0 * s.val, s.b, x) <= 1.0000001e-10
    A.drop_csr()
    x2, r2 = bicgstab(ctx, A, s.b, rtol=1e-10, loop=loop)
    assert np.array_equal(x, x2)
    A.close()


def test_fixed_iterations(ctx):
    s = synth.convdiff2d(60, 30.0, seed=2)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    x, r = bicgstab(ctx, A, s.b, rtol=0.0, maxit=12, fixed_iters=True)
    ref = orc.bicgstab_fixed(s.rowptr, s.col, s.val, s.b, np.zeros(s.n), 12)[0]
    assert r.iters == 12 and r.status == 0
    assert np.max(np.abs(x - ref)) <= 1e-10 * np.max(np.abs(ref))
    A.close()


@pytest.mark.parametrize("m", [500, 20_000, 40_001])
@pytest.mark.parametrize("loop", ["merged", "classic"])
def test_infinite_entry(ctx, m, loop):
    """From x0 = 0 the residual is b whatever A holds, so the iterate stays 0; from another x0 it is not finite."""
    rp, col, val = _dominant(m, 4, m)
    val[rp[m // 2]] = np.inf
    b = np.random.default_rng(m).standard_normal(m)
    A = Matrix.from_csr(ctx, rp, col, val)
    x, r = bicgstab(ctx, A, b, rtol=1e-10, loop=loop, raise_on_error=False)
    assert r.status == 5 and r.iters == 0 and np.array_equal(x, np.zeros(m))
    x, r = bicgstab(ctx, A, b, np.ones(m), rtol=1e-10, loop=loop, raise_on_error=False)
    assert r.status == 5 and r.iters == 0 and np.array_equal(x, np.ones(m))
    A.close()
