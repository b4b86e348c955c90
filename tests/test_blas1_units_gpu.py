"""BLAS-1 at the edges of the kernels' units (2 elements) and batches, on vectors at either 8-byte
alignment: the result does not depend on it; nothing past the end is touched."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 3, 255, 512, 513, 1023, 77_823, 155_649, 311_297, 700_001, 1_245_185]


def _at(v, off):
    """v on the device, `off` doubles behind a 16-byte boundary, inside a buffer of sevens."""
    buf = torch.full((v.size + 4,), 7.0, dtype=torch.float64, device="cuda")
    view = buf[off:off + v.size]
    view.copy_(dev(v))
    return buf, view


@pytest.mark.parametrize("n", SIZES)
def test_units_and_alignment(ctx, n):
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal(n), rng.standard_normal(n)
    bound = 1e-14 * float(np.sum(np.abs(x * y)))
    first = None
    for ox, oy in ((0, 0), (0, 1), (1, 0), (1, 1)):
        bx, xd = _at(x, ox)
        by, yd = _at(y, oy)
        d = ctx.dot(xd, yd)
        assert abs(d - orc.dot(x, y)) <= bound
        first = d if first is None else first
        assert d == first
        ctx.axpy(-0.3751, xd, yd)
        # one fused multiply-add: within an ulp of the separately rounded value's neighbourhood
        want = -0.3751 * x + y
        assert np.all(np.abs(yd.cpu().numpy() - want) <= 2.3e-16 * (np.abs(0.3751 * x) + np.abs(want)))
        ctx.scal(2.5, xd)
        assert np.array_equal(xd.cpu().numpy(), 2.5 * x)
        for buf, off in ((bx, ox), (by, oy)):
            rest = torch.cat([buf[:off], buf[off + n:]])
            assert torch.all(rest == 7.0)


def test_axpy_onto_itself(ctx):
    x = np.random.default_rng(3).standard_normal(100_003)
    xd = dev(x)
    ctx.axpy(0.5, xd, xd)
    assert np.array_equal(xd.cpu().numpy(), 1.5 * x)
