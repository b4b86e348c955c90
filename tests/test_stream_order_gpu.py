"""Calls on device tensors are ordered with torch's current stream both ways: late inputs on a side
stream, results read there at once, several streams in turn on one context, and stream capture."""
import numpy as np
import pytest
import torch

from gpu_util import dev
from hethyppar_gb300 import Matrix, synth
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_side_streams_in_turn(ctx):
    s = synth.convdiff2d(300, 20.0)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    rng = np.random.default_rng(0)
    xs = [rng.standard_normal(s.n) for _ in range(4)]
    src = [dev(x) for x in xs]
    x, y = torch.zeros(s.n, dtype=torch.float64, device="cuda"), torch.zeros(s.n, dtype=torch.float64, device="cuda")
    out = [torch.empty_like(y) for _ in xs]
    A.spmv_dev(x, y)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    prev = streams[1]
    for st, v, o in zip(streams, src, out):
        st.wait_stream(prev)
        with torch.cuda.stream(st):
            torch.cuda._sleep(2_000_000)  # x is written a millisecond after the call is queued
            x.copy_(v)
            A.spmv_dev(x, y)
            x.zero_()  # only after the product has read it
            o.copy_(y)
        prev = st
    torch.cuda.synchronize()
    for xh, o in zip(xs, out):
        assert np.array_equal(o.cpu().numpy(), orc.spmv(s.rowptr, s.col, s.val, xh, fma=True))
    A.close()


def test_under_capture(ctx):
    s = synth.convdiff2d(100, 20.0)
    A = Matrix.from_csr(ctx, s.rowptr, s.col, s.val)
    x = dev(np.random.default_rng(1).standard_normal(s.n))
    y, d = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")

    def step():
        A.spmv_dev(x, y)
        ctx.axpy(0.5, x, y)
        ctx.dot(x, y, out=d)

    step()  # layout and scratch
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        step()
    for k in range(3):
        x.mul_(1.0 + k)
        step()
        want_y, want_d = y.clone(), d.clone()
        y.zero_()
        d.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want_y) and torch.equal(d, want_d)
    A.close()
