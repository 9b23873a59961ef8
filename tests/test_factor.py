"""The DIC / DILU factor of the one-launch sweeps at the edges of its range."""
import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300 import _lib
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
