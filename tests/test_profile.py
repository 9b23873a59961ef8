"""fcg_profile_sweeps times the kernels that the last solve ran."""
import os

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from tests.meshes import poisson_system
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu

LOOP = ["k_cg_p", "k_cg_spmv", "k_cg_update"]


@pytest.mark.parametrize("ext,units", [((12, 9, 7), ["k_resident_dpcg"]),
                                       ((67, 67, 67), ["k_resident_dpcg"]), ((68, 68, 68), LOOP)])
def test_profiled_kernels_are_those_of_the_solve(ext, units):
    m = box_mesh(*ext)
    c = fcg.Context(m)
    a, su = c.laplacian(*poisson_system(m))
    zero = np.zeros(m.numCells)
    r = c.dpcg(a, su, zero, 1e-30, 20)
    ms = c.profile_sweeps(5)
    assert list(ms) == units and all(v > 0 for v in ms.values())
    assert np.array_equal(c.dpcg(a, su, zero, 1e-30, 20).fi, r.fi)
    os.environ["FCG_NO_GRAPH"] = "1"  # the loop, whatever the size
    try:
        c.dpcg(a, su, zero, 1e-30, 20)
        assert list(c.profile_sweeps(5)) == LOOP
    finally:
        del os.environ["FCG_NO_GRAPH"]
    c.iccg(a, su, zero, 1e-30, 4)
    assert list(c.profile_sweeps(2))[:2] == ["fwd_levels", "bwd_levels"]
    c.close()
