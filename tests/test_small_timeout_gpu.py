"""A wait of the one-kernel solves that runs out: with a limit of no reads at all, every block gives up in the
first exchange. The solve reports it, and the context and the matrix go on."""
import numpy as np
import pytest
import torch

from hethyppar_gb300 import HHPError, Matrix, bicgstab, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
TIMEOUT = 7  # HHP_ERR_TIMEOUT


@pytest.fixture
def timed_out(ctx, monkeypatch):
    """A system of the grid form, after a solve whose wait ran out."""
    s = synth.convdiff2d(100, 30.0, seed=1)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    monkeypatch.setenv("HHP_SOLVE_GRAPH", "0")  # a graph would keep the limit it was captured with
    monkeypatch.setenv("HHP_SMALL_POLLS", "0")
    with pytest.raises(HHPError) as e:
        bicgstab(ctx, A, s.b, rtol=1e-10)
    monkeypatch.delenv("HHP_SMALL_POLLS")
    yield s, A, e.value
    A.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_reported_and_over(ctx, monkeypatch, timed_out, precision):
    s, A, error = timed_out
    assert error.status == TIMEOUT and "one-kernel solve" in str(error) and "SpMV" not in str(error)
    monkeypatch.setenv("HHP_SMALL_POLLS", "0")
    _, r = bicgstab(ctx, A, s.b, rtol=1e-10, precision=precision, raise_on_error=False)
    assert r.status == TIMEOUT
    monkeypatch.delenv("HHP_SMALL_POLLS")
    for graph in ("0", "1"):
        monkeypatch.setenv("HHP_SOLVE_GRAPH", graph)
        x, r = bicgstab(ctx, A, s.b, rtol=1e-10, precision=precision)
        d = s.b - orc.spmv(s.rowptr, s.col, s.val, x)
        assert r.status == 0 and np.sqrt(orc.dot(d, d) / orc.dot(s.b, s.b)) <= 1.0000001e-10


def test_products_after_it_are_computed(ctx, timed_out):
    """The error that the solve has reported does not stop what the caller launches next."""
    s, A, _ = timed_out
    x = torch.as_tensor(np.random.default_rng(3).standard_normal(s.n)).cuda()
    y, z = torch.zeros_like(x), torch.zeros_like(x)
    A.spmv_dev(x, y)
    A.spmv_t_dev(x, z)
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), orc.spmv(s.rowptr, s.col, s.val, x.cpu().numpy(), fma=True))
    tr, tc, tv = orc.csr_to_csc(s.rowptr, s.col, s.val, s.n)
    assert np.array_equal(z.cpu().numpy(), orc.spmv(tr, tc, tv, x.cpu().numpy(), fma=True))
