"""Batches of many small systems: the lanes that close a system's sums at every number of
systems where their number changes, against the solver of one system."""
import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from tests.meshes import poisson_system
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsys", [1, 8, 9, 16, 17, 32, 33, 64])
def test_batch_of_many_systems_matches_single_solves(nsys):
    """Uneven systems, so that some stop while others go on. The recurrence is that of
    fcg_dpcg; the sums are added in another order, an ulp a sweep: 1e-10, as the other
    solvers' comparisons ask, and a sweep more or less at the stop test."""
    ctx, a, su = [], [], []
    for k in range(nsys):
        m = box_mesh(3 + k % 5, 4 + k % 7, 5 + k % 3, seed=k)
        c = fcg.Context(m)
        x = c.laplacian(*poisson_system(m, seed=k + 1))
        ctx.append(c)
        a.append(x[0])
        su.append(x[1])
    b = fcg.Batch(ctx)
    zero = [np.zeros(c.n) for c in ctx]
    for sor, nsw in ((1e-30, 8), (1e-9, 400)):
        fi, rep = b.dpcg(a, su, zero, sor, nsw)
        for k in range(nsys):
            o = ctx[k].dpcg(a[k], su[k], zero[k], sor, nsw)
            assert abs(rep[k].iters - o.iters) <= (0 if nsw == 8 else 1)
            assert rep[k].converged == o.converged
            tol = 1e-10 if nsw == 8 else 1e-8
            assert np.abs(fi[k] - o.fi).max() <= tol * np.abs(o.fi).max(), k
        again, _ = b.dpcg(a, su, zero, sor, nsw)
        assert all(np.array_equal(x, y) for x, y in zip(fi, again))
    b.close()
    for c in ctx:
        c.close()
