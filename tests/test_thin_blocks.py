"""Thin hex blocks, whose wavefront records would hold many times their cells: level order
where the tiles are many, the wavefront form where they are few, with the same bits."""
import os

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300.systems import transport_systems
from tests.meshes import poisson_system
from tests.test_wave_blocks import _context, box_mesh

pytestmark = pytest.mark.gpu


def test_sweeps_of_a_thin_block_take_memory_by_its_cells():
    """Two planes of 640 x 640 cells. The arrays in level order are 4 values and, for three
    entries a triangle, 6 coefficients and 12 indices a cell, with positions and padding about
    200 bytes; the wavefront form's 10 values for each of 12 positions a cell are 960 (FP32:
    480 a system)."""
    torch = pytest.importorskip("torch")
    m = box_mesh(640, 640, 2)
    c = fcg.Context(m)
    a, su = c.laplacian(*poisson_system(m))
    zero = np.zeros(m.numCells)
    A, S, _ = transport_systems(m, c.create_csr(), nsys=2)
    c.dpcg(a, su, zero, 0.0, 2)  # the solvers' common state and staging

    def growth(fn):
        before = torch.cuda.mem_get_info()[0]
        fn()
        return (before - torch.cuda.mem_get_info()[0]) / m.numCells

    assert growth(lambda: c.iccg(a, su, zero, 0.0, 2)) < 400
    # values, 12 vectors and the staging of two systems: 7 (8 + 4) + 4 7 + 8 (3 + 5) + 8 (7 + 2)
    # = 250 bytes a cell and system, and half the sweeps' of FP64
    assert growth(lambda: c.bicgstab_multi(A, S, np.zeros_like(S), 1e-6, 2)) < 800
    c.close()


@pytest.mark.parametrize("dims", [(37 * 16, 65 * 8, 2), (2, 300, 200), (640, 640, 2)])
def test_thin_blocks_have_the_bits_of_the_level_order(dims):
    """Just below the number of tiles that goes over to level order, two cells in i, and past
    the line."""
    m = box_mesh(*dims)
    ctxs = [_context(m), _context(m, "rows")]
    a, su = ctxs[0].laplacian(*poisson_system(m))
    A, S, _ = transport_systems(m, ctxs[0].create_csr(), nsys=2)
    x0 = np.zeros(m.numCells)
    for solver in ("iccg", "bicgstab"):
        r, o = [getattr(c, solver)(a, su, x0, 0.0, 4) for c in ctxs]
        assert np.array_equal(r.fi, o.fi) and r.resl == o.resl
    x = []
    for c, mode in zip(ctxs, (None, "rows")):
        saved = os.environ.pop("FCG_SWEEP", None)
        if mode:
            os.environ["FCG_SWEEP"] = mode  # read when the multi-RHS state is made
        try:
            x.append(c.bicgstab_multi(A, S, np.zeros_like(S), 1e-8, 100)[0])
        finally:
            os.environ.pop("FCG_SWEEP", None)
            if saved is not None:
                os.environ["FCG_SWEEP"] = saved
        c.close()
    assert np.array_equal(*x)
