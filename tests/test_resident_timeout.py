"""The bounded waits of the resident DPCG: a block that gives up on a sum and leaves without
storing its rows makes the solve return FCG_ERR_TIMEOUT, also when every other block saw
the sum complete, and the context then solves normally."""
import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300 import _lib
from tests.meshes import poisson_system
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ext,row", [((24, 24, 24), 13824), ((24, 24, 24), 1), ((43, 43, 43), 30000),
                                     ((5, 3, 2), 7)])
@pytest.mark.parametrize("nsw", [1, 2, 40])
def test_a_block_that_gives_up_ends_the_solve_with_a_timeout(ext, row, nsw):
    """nsw = 1: the block gives up on the last sum of the solve, which the others pass, block 0
    among them for the rows past its own.  More sweeps: the others wait for the block that
    left.  One block alone (30 rows) gives up on its own sum."""
    m = box_mesh(*ext)
    c = fcg.Context(m)
    a, su = c.laplacian(*poisson_system(m))
    fi = fcg.uniform(3, 1, m.numCells)
    before = c.dpcg(a, su, fi, 1e-30, min(nsw, 15))
    c.set_sweep_wait_test(polls=4096, absent_row=row)
    with pytest.raises(_lib.FcgError) as ei:
        c.dpcg(a, su, fi, 1e-30, nsw)
    assert ei.value.status == _lib.FCG_ERR_TIMEOUT and "wait gave up" in str(ei.value)
    c.set_sweep_wait_test(0, 0)
    after = c.dpcg(a, su, fi, 1e-30, min(nsw, 15))
    assert np.array_equal(before.fi, after.fi) and np.array_equal(before.res, after.res)
    c.close()
