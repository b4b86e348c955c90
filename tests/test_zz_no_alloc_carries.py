"""hhp_spmv_csr_noalloc on rows that span many CTAs: the carries of a row's run are added by one warp, whatever
the run's length is to its 32 lanes and 128 requests, and a long row does not wait for them one by one."""
import ctypes

import numpy as np
import pytest
import torch

from hethyppar_gb300 import _lib
from test_zz_no_alloc import _case

pytestmark = pytest.mark.gpu
ITEMS = 512  # rows + nonzeros of a CTA on short lists


def _csr(lens, n, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return rp, rng.integers(0, n, size=int(rp[-1])).astype(np.int32), rng.standard_normal(int(rp[-1]))


@pytest.mark.parametrize("ctas", [1, 2, 3, 31, 32, 33, 64, 127, 128, 129, 160, 161, 257, 700])
@pytest.mark.parametrize("around", [[], [3, 0, 17], [900, 1]])
def test_runs(ctx, ctas, around):
    n = 10_001
    lens = around + [ITEMS * ctas - 1 - sum(around) // 2] + around[::-1]
    rp, col, val = _csr(lens, n, ctas)
    _case(ctx, rp, col, val, n, alpha=1.0, beta=0.0, seed=1)
    _case(ctx, rp, col, val, n, alpha=-0.75, beta=2.0, seed=2)
    rp, col, val = _csr(lens * 3, n, ctas)  # several runs one after another
    _case(ctx, rp, col, val, n, alpha=0.5, beta=1.0, seed=3)


def test_one_row_takes_no_longer_than_its_entries():
    """777,777 entries in one row (12 us) against the same number in rows of 1000; with its 760 carries added one
    after another the row took 107 us."""
    n, us = 100_000, []
    for lens in ([1000] * 777 + [777], [777_777]):
        rp, col, val = _csr(lens, n, 0)
        rp, col, val = (torch.as_tensor(a).cuda() for a in (rp, col, val))
        x, y = torch.ones(n, dtype=torch.float64, device="cuda"), torch.zeros(len(lens), dtype=torch.float64, device="cuda")
        args = [len(lens), n, 777_777, *(ctypes.c_void_p(t.data_ptr()) for t in (rp, col, val)), 1.0,
                ctypes.c_void_p(x.data_ptr()), 0.0, ctypes.c_void_p(y.data_ptr()),
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)]
        for _ in range(3):
            _lib.check(_lib.lib().hhp_spmv_csr_noalloc(*args), "hhp_spmv_csr_noalloc")
        times = []
        for _ in range(7):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(20):
                _lib.lib().hhp_spmv_csr_noalloc(*args)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b) * 50.0)
        us.append(float(np.median(times)))
    assert us[1] < 3.0 * us[0], us
