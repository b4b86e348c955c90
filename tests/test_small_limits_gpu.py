"""One-kernel solves of several systems side by side: what one system needs of shared memory must not limit
another's later launches, in one context, in two, and from two threads."""
import math
import threading

import numpy as np
import pytest

from hethyppar_gb300 import Context, Matrix, bicgstab, synth
from oracle import oracle as orc
from test_small_solve_gpu import _dominant

pytestmark = pytest.mark.gpu

# the first system's blocks hold several times the entries of the second's (cluster form, then grid form)
PAIRS = [((5000, 16), 64), ((20_000, 31), 100)]
CALLS = [dict(loop=loop, precision=precision) for precision in ("fp64", "mixed") for loop in ("merged", "classic")]


def _systems(pair):
    (m, width), n = pair
    rp, col, val = _dominant(m, width, m)
    s = synth.convdiff2d(n, 30.0, seed=1)
    return [(rp, col, val, np.random.default_rng(m).standard_normal(m)), (s.rowptr, s.col, s.val, s.b)]


def _check(ctx, A, system, **kw):
    rp, col, val, b = system
    x, r = bicgstab(ctx, A, b, rtol=1e-10, **kw)
    d = b - orc.spmv(rp, col, val, x)
    assert r.status == 0 and math.sqrt(orc.dot(d, d) / orc.dot(b, b)) <= 1.0000001e-10


@pytest.mark.parametrize("pair", PAIRS)
@pytest.mark.parametrize("graph", ["1", "0"])
def test_two_systems_in_turn(ctx, monkeypatch, pair, graph):
    monkeypatch.setenv("HHP_SOLVE_GRAPH", graph)
    big, little = _systems(pair)
    A, B = Matrix.from_csr(ctx, *big[:3]), Matrix.from_csr(ctx, *little[:3])
    _check(ctx, A, big)
    _check(ctx, B, little)
    for kw in CALLS:  # each a launch of its own that the second system's set-up came before
        _check(ctx, A, big, **kw)
        _check(ctx, B, little, **kw)
    x, r = bicgstab(ctx, A, big[3], rtol=0.0, maxit=5, fixed_iters=True)
    assert r.status == 0 and r.iters == 5
    A.close()
    B.close()


def _together(systems):
    """Every call for each of the systems, a context and a thread each."""
    failed = []

    def work(system):
        try:
            with Context(0) as c:
                for kw in CALLS * 3:
                    A = Matrix.from_csr(c, *system[:3])
                    _check(c, A, system, **kw)
                    A.close()
        except BaseException as e:  # noqa: BLE001 -- reported by the test's own thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in systems]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed


@pytest.mark.parametrize("pair", PAIRS)
def test_two_contexts_on_two_threads(pair):
    _together(_systems(pair))


def test_two_grids_that_do_not_fit_together():
    """One block of either takes more than half of an SM's shared memory: one solve's grid waits for the other's."""
    m, width = 20_000, 62
    _together([(*_dominant(m, width, seed), np.random.default_rng(seed).standard_normal(m)) for seed in (1, 2)])
