"""The two-colour ILU(0) application (a warp per slice, two passes) where its layout can go wrong:
rows just at and around the 32-row slices, several widths per level, more widths than it takes,
columns whose distance from the row does and does not fit 16 bits, rows beyond its length limit.
Bit for bit against the oracle, out of place and in place, before and after new values."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from hethyppar_gb300 import Matrix, bicgstab, reorder_color, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _bipartite(half_a, half_b, lens, spread, seed):
    """Rows 0..half_a-1 couple only to rows half_a.. and the other way round (symmetric pattern):
    row i of the first colour has lens[i mod len(lens)] neighbours within `spread` of its place."""
    rng = np.random.default_rng(seed)
    m = half_a + half_b
    nb = [set() for _ in range(m)]
    for i in range(half_a):
        centre = i * half_b // half_a
        for _ in range(lens[i % len(lens)]):
            j = half_a + int(np.clip(centre + rng.integers(-spread, spread + 1), 0, half_b - 1))
            nb[i].add(j)
            nb[j].add(i)
    for i in range(m):  # nobody alone: a row without neighbours is on level 0 of both triangles
        if not nb[i]:
            j = half_a if i < half_a else 0
            nb[i].add(j)
            nb[j].add(i)
    cols = [sorted(n | {i}) for i, n in enumerate(nb)]
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = rng.uniform(-1.0, 0.0, col.size)
    rows = np.repeat(np.arange(m), np.diff(rp))
    diag = col == rows
    val[diag] = 1.0 + np.bincount(rows, weights=np.abs(val * ~diag), minlength=m)
    return rp, col, val


def _stencil(dims):
    rp, col, val = synth._stencil(dims, 20.0, (1.0, 0.5, 0.25)[:len(dims)])
    perm, nc = reorder_color(rp, col)
    assert nc == 2
    rp, col, val = orc.csr_permute(rp, col, val, perm)
    order = np.concatenate([np.argsort(col[a:b], kind="stable") + a for a, b in zip(rp[:-1], rp[1:])])
    return rp, col[order], val[order]


CASES = {
    "2x1": lambda: _bipartite(1, 1, [1], 0, 1),
    "31+33": lambda: _bipartite(31, 33, [1, 2, 3], 4, 2),
    "32+32": lambda: _bipartite(32, 32, [4], 9, 3),
    "10x10": lambda: _stencil((10, 10)), "65x64": lambda: _stencil((65, 64)), "12^3": lambda: _stencil((12, 12, 12)),
    "33x32x31": lambda: _stencil((33, 32, 31)),
    "far_columns": lambda: _bipartite(50_000, 90_000, [2, 5], 80_000, 4),   # distances over 16 bits
    "many_widths": lambda: _bipartite(2_000, 2_000, list(range(1, 30)), 700, 5),  # more than 8 runs
    "long_rows": lambda: _bipartite(300, 4_000, [3, 90], 2_000, 6),         # over 64 entries: warp-summed
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_two_colour_application(ctx, name):
    rp, col, val = CASES[name]()
    m = rp.size - 1
    A = Matrix.from_csr(ctx, rp, col, val)
    _, levels = A.ilu0_factor()
    assert levels == (2, 2)
    st, lu, _ = orc.ilu0(rp, col, val)
    assert st == 0
    rng = np.random.default_rng(7)
    for _ in range(2):
        r = rng.standard_normal(m)
        ref = orc.ilu0_apply(rp, col, lu, r)
        rd, z = dev(r), torch.full((m,), float("nan"), dtype=torch.float64, device="cuda")
        A.ilu0_apply_dev(rd, z)
        assert np.array_equal(z.cpu().numpy(), ref)
        A.ilu0_apply_dev(rd, rd)
        assert np.array_equal(rd.cpu().numpy(), ref)
    b = rng.standard_normal(m)
    x, res = bicgstab(ctx, A, b, rtol=1e-10, maxit=500, precond="ilu0")
    assert res.status == 0
    resid = b - orc.spmv(rp, col, val, x)
    assert np.sqrt(orc.dot(resid, resid) / orc.dot(b, b)) <= 1.0000001e-10
    # new values: the factors and the layout are built again
    A.set_values(2.0 * val)
    z = torch.empty(m, dtype=torch.float64, device="cuda")
    A.ilu0_apply_dev(dev(b), z)
    assert np.array_equal(z.cpu().numpy(), orc.ilu0_apply(rp, col, orc.ilu0(rp, col, 2.0 * val)[1], b))
    A.close()
