"""The DIC / DILU factor of the one-launch sweeps at the edges of its range."""
import os

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300 import _lib
from freecappuccino_gb300.systems import transport_systems
from tests.meshes import poisson_system
from tests.test_wave_blocks import _context, box_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [None, "rows"])
@pytest.mark.parametrize("solver", ["iccg", "bicgstab", "dpcg_mixed"])
def test_broken_pivot_is_reported_when_no_sweep_is_due(mode, solver):
    """No sweep allowed, or a first residual below the early-exit tolerance: the factor's
    breakdown is reported all the same, in wavefront and in level order."""
    m = box_mesh(12, 9, 7)
    c = _context(m, mode)
    a, su = c.laplacian(*poisson_system(m))
    diag = c.create_csr()[2] - 1
    bad = a.copy()  # rows 0 and 1: 4, 2 and 2, 1, so that the second pivot is 1 - 2 (2 / 4)
    bad[diag[0]:diag[0] + 2] = 4.0, 2.0
    bad[diag[1] - 1:diag[1] + 1] = 2.0, 1.0
    zero = np.zeros(m.numCells)
    for rhs, nsw in ((su, 0), (zero, 10)):
        assert getattr(c, solver)(a, rhs, zero, 1e-8, nsw).iters == 0
        with pytest.raises(_lib.FcgError) as ei:
            getattr(c, solver)(bad, rhs, zero, 1e-8, nsw)
        assert ei.value.status == _lib.FCG_ERR_PIVOT
    assert getattr(c, solver)(a, su, zero, 1e-8, 2000).converged
    c.close()


@pytest.mark.parametrize("mode", [None, "rows", "levels"])
@pytest.mark.parametrize("powers", [(-80,), (0, -80, 20), (-90, 10)])
def test_multi_rhs_factor_does_not_depend_on_the_systems_scale(mode, powers):
    """A matrix times a power of two has the solution over that power, and every operation of
    the solver, FP32 ones included, the same digits, as long as none leaves the range: the
    products of two coefficients near 2^-80 would."""
    m = box_mesh(17, 9, 4)
    saved = os.environ.pop("FCG_SWEEP", None)
    if mode:
        os.environ["FCG_SWEEP"] = mode  # read when the multi-RHS state is made
    try:
        c = fcg.Context(m)
        a, su, _ = transport_systems(m, c.create_csr(), nsys=len(powers))
        want, wr = c.bicgstab_multi(a, su, np.zeros_like(su), 1e-10, 200)
        s = 2.0 ** np.array(powers, float)[:, None]
        got, gr = c.bicgstab_multi(a * s, su, np.zeros_like(su), 1e-10, 200)
    finally:
        os.environ.pop("FCG_SWEEP", None)
        if saved is not None:
            os.environ["FCG_SWEEP"] = saved
    c.close()
    assert np.array_equal(got * s, want)
    assert [r.iters for r in gr] == [r.iters for r in wr] and all(r.converged for r in gr)


@pytest.mark.parametrize("mode", [None, "rows"])
def test_multi_rhs_factor_of_large_coefficients(mode):
    """Coefficients whose products overflow FP32, themselves far from it."""
    m = box_mesh(17, 9, 4)
    saved = os.environ.pop("FCG_SWEEP", None)
    if mode:
        os.environ["FCG_SWEEP"] = mode
    try:
        c = fcg.Context(m)
        a, su, _ = transport_systems(m, c.create_csr(), nsys=2)
        big = 1e22 / np.abs(a).max()
        _, rep = c.bicgstab_multi(a * big, su, np.zeros_like(su), 1e-10, 200)
    finally:
        os.environ.pop("FCG_SWEEP", None)
        if saved is not None:
            os.environ["FCG_SWEEP"] = saved
    c.close()
    assert all(r.converged for r in rep)
