"""The DPCG whose rows stay in the resident threads against the captured loop's kernels, at
the edges of the sizes each takes."""
import os

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from tests.meshes import poisson_system
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu


def _host_driven(fn):
    """fn() with the loop of separate kernels, driven from the host."""
    os.environ["FCG_NO_GRAPH"] = "1"
    try:
        return fn()
    finally:
        del os.environ["FCG_NO_GRAPH"]


# one slice and less, ragged slices, the largest system of one, two and four rows a thread on
# 152 SMs and the next ones; 68^3 is past them all
@pytest.mark.parametrize("ext", [(2, 1, 1), (5, 3, 2), (11, 3, 1), (24, 24, 24), (47, 41, 40),
                                 (43, 43, 43), (60, 51, 51), (67, 67, 67), (68, 68, 68)])
def test_resident_dpcg_matches_the_loop(ext):
    """Both round a row's sums alike up to the direction formed on the fly and add the blocks'
    partial sums in another order, an ulp of each sum a sweep: 1e-10 after 25 sweeps, as the
    oracle's own comparison asks.  The trace is that of the stop test."""
    m = box_mesh(*ext)
    c = fcg.Context(m)
    a, su = c.laplacian(*poisson_system(m))
    fi = fcg.uniform(3, 1, m.numCells)
    for nsw in sorted({0, 1, min(2, m.numCells // 2), min(25, m.numCells // 2)}):
        r = c.dpcg(a, su, fi, 1e-30, nsw, want_trace=True)
        o = _host_driven(lambda: c.dpcg(a, su, fi, 1e-30, nsw, want_trace=True))
        again = c.dpcg(a, su, fi, 1e-30, nsw)
        assert r.iters == o.iters == nsw and r.converged == o.converged
        assert np.array_equal(r.fi, again.fi) and np.array_equal(r.res, again.res)
        tr, to = np.asarray(r.trace)[:nsw], np.asarray(o.trace)[:nsw]
        r0 = r.res0
        assert abs(r.res0 - o.res0) <= 1e-10 * r0
        for x, y, scale in ((r.fi, o.fi, np.abs(o.fi).max()), (r.res, o.res, r0),
                            (tr[:, 0], to[:, 0], r0), (tr[:, 1], to[:, 1], 1.0)):
            assert np.abs(x - y).max(initial=0.0) <= 1e-10 * scale
    c.close()


def test_resident_dpcg_stops_and_fails_as_the_loop():
    m = box_mesh(12, 9, 7)
    c = fcg.Context(m)
    a, su = c.laplacian(*poisson_system(m))
    zero = np.zeros(m.numCells)
    r = c.dpcg(a, su, zero, 1e-6, 500)
    o = _host_driven(lambda: c.dpcg(a, su, zero, 1e-6, 500))
    assert r.converged and o.converged and abs(r.iters - o.iters) <= 1 and r.iters < 500
    assert c.dpcg(a, zero, zero, 1e-6, 500).iters == 0  # below the early-exit tolerance
    bad = su.copy()
    bad[5] = np.nan
    for run in (lambda f: f(), _host_driven):
        with pytest.raises(fcg._lib.FcgError, match="non-finite"):
            run(lambda: c.dpcg(a, bad, zero, 1e-6, 10))
    assert c.dpcg(a, su, zero, 1e-6, 500).iters == r.iters  # the state is usable afterwards
    c.close()


def test_resident_dpcg_of_two_threads():
    """Two contexts, each in its own thread and stream, solve at the same time: the launches
    are cooperative, so the blocks of one never wait for blocks that cannot run."""
    import threading

    ctx, sys_, ref = [], [], []
    for ext in ((24, 24, 24), (43, 43, 43)):
        m = box_mesh(*ext)
        c = fcg.Context(m)
        a, su = c.laplacian(*poisson_system(m))
        ctx.append(c)
        sys_.append((a, su, np.zeros(m.numCells)))
        ref.append(c.dpcg(*sys_[-1], 1e-30, 25).fi)
    bad = []

    def run(k):
        for _ in range(20):
            if not np.array_equal(ctx[k].dpcg(*sys_[k], 1e-30, 25).fi, ref[k]):
                bad.append(k)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for c in ctx:
        c.close()
