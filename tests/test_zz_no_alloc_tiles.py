"""hhp_spmv_csr_noalloc at the edges of its tiles: row counts and lengths around the tile size (1664
merge items), the lane-per-row limit (longest row x rounds of 128 rows = 48), empty rows, rows over
several tiles and CTAs, lists below one CTA's minimum; and under stream capture."""
import ctypes

import numpy as np
import pytest
import torch

from hethyppar_gb300 import _lib
from test_zz_no_alloc import _case, _noalloc

SHAPES = [
    ("tiny", [0]), ("tiny2", [3, 0, 1]), ("one_tile", [12] * 128), ("one_tile_over", [12] * 129),
    ("len48", [48] * 4001), ("len49", [49] * 4001), ("two_rounds_24", [24, 0, 1] * 30_000),
    ("empty", [0] * 50_000), ("ones", [1] * 300_001), ("len17", [17] * 60_013), ("len1663", [1663] * 700),
    ("len1664", [1664] * 700), ("len5000", [5000] * 301), ("one_row", [777_777]),
    ("mixed", ([17] * 997 + [0] * 500 + [300] + [2] * 1501 + [70_000]) * 5),
]


@pytest.mark.gpu
@pytest.mark.parametrize("name,lens", SHAPES, ids=[s[0] for s in SHAPES])
def test_noalloc_tile_edges(ctx, name, lens):
    rng = np.random.default_rng(len(lens))
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n = 70_001
    col = rng.integers(0, n, size=int(rp[-1])).astype(np.int32)
    val = rng.standard_normal(int(rp[-1]))
    if rp[-1] == 0:  # nothing stored: y = beta y
        y0 = rng.standard_normal(rp.size - 1)
        col, val = np.zeros(1, np.int32), np.zeros(1)
        assert np.array_equal(_noalloc(rp, col, val, np.ones(n), 2.0, 0.5, y0, n), 0.5 * y0)
        return
    _case(ctx, rp, col, val, n, alpha=1.0, beta=0.0, seed=7)
    _case(ctx, rp, col, val, n, alpha=-0.75, beta=2.0, seed=8)
    # beta = 0 does not read y
    x = rng.standard_normal(n)
    a = _noalloc(rp, col, val, x, 1.0, 0.0, np.full(rp.size - 1, np.nan), n)
    assert np.array_equal(a, _noalloc(rp, col, val, x, 1.0, 0.0, np.zeros(rp.size - 1), n))


@pytest.mark.gpu
def test_noalloc_under_capture(ctx):
    rng = np.random.default_rng(0)
    lens = np.full(20_000, 17)
    lens[777] = 90_000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    m = n = lens.size
    col = torch.from_numpy(rng.integers(0, n, size=int(rp[-1])).astype(np.int32)).cuda()
    val, x = torch.randn(int(rp[-1]), dtype=torch.float64).cuda(), torch.randn(n, dtype=torch.float64).cuda()
    d_rp, y, z = torch.from_numpy(rp).cuda(), torch.empty(m, dtype=torch.float64).cuda(), torch.empty(m, dtype=torch.float64).cuda()

    def call(out):
        s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert _lib.lib().hhp_spmv_csr_noalloc(m, n, int(rp[-1]), d_rp.data_ptr(), col.data_ptr(), val.data_ptr(), 1.0,
                                               x.data_ptr(), 0.0, out.data_ptr(), s) == 0

    call(y)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(z)
    for _ in range(3):
        z.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, z)
