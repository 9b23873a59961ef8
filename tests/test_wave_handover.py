"""Hand-over of the wavefront-tiled sweeps between blocks: nothing is stored into another
block's shared memory before the cluster has started, and clusters that wait on one another
over more planes than one launch takes."""
import os
import re

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300 import _lib
from tests.meshes import poisson_system
from tests.test_wave_blocks import _context, box_mesh

CSRC = os.path.join(os.path.dirname(fcg.__file__), "csrc")


def test_no_access_to_a_peer_block_before_the_cluster_has_started():
    """The programming model lets a block touch another's shared memory once every block of
    the cluster has started, which the first cluster-wide barrier tells.  No run shows a
    breach of it reliably, so the kernel's source is read: from its first line to its first
    wait for the cluster there is no address of a peer and no access through one."""
    src = open(os.path.join(CSRC, "wave_sweep.cuh")).read()
    src = re.sub(r"//[^\n]*", "", src)
    body = src[src.index("k_wave_sweep(int nx"):]
    body = body[:body.index("for_cells(")]
    first = min(m.start() for m in re.finditer(r"cluster\.(sync|barrier_wait)\(\)", body))
    uses = [m.start() for m in re.finditer(r"peer_addr|shared::cluster|W::push|map_shared_rank", body)]
    assert uses and min(uses) > first


@pytest.fixture(scope="module")
def tall():
    """Two by two clusters of 32 x 32 columns, 513 planes: two launches a sweep."""
    return box_mesh(35, 37, 513)


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["iccg", "bicgstab"])
def test_clusters_hand_over_in_every_slab(tall, solver):
    """The rounding of a row is that of the level-ordered form: the same bits.  Solved twice:
    the second solve finds sentinels and counters as the first left them."""
    ctxs = [_context(tall), _context(tall, "rows")]
    mu, phi, su0 = poisson_system(tall)
    a, su = ctxs[0].laplacian(mu, phi, su0)
    x0 = np.zeros(tall.numCells)
    for _ in range(2):
        r, o = [getattr(c, solver)(a, su, x0, 0.0, 6) for c in ctxs]
        assert np.array_equal(r.fi, o.fi) and r.resl == o.resl
    for c in ctxs:
        c.close()


@pytest.mark.gpu
def test_clusters_hand_over_in_every_slab_multi_rhs(tall):
    """The FP32 form, three systems in one launch."""
    from freecappuccino_gb300.systems import transport_systems

    out = []
    for mode in (None, "rows"):
        c = fcg.Context(tall)
        a, su, _ = transport_systems(tall, c.create_csr(), nsys=3)
        saved = os.environ.pop("FCG_SWEEP", None)
        if mode:
            os.environ["FCG_SWEEP"] = mode  # read when the multi-RHS state is made
        try:
            out.append([c.bicgstab_multi(a, su, np.zeros_like(su), 1e-10, 200)
                        for _ in range(2)][1])
        finally:
            os.environ.pop("FCG_SWEEP", None)
            if saved is not None:
                os.environ["FCG_SWEEP"] = saved
        c.close()
    (x1, r1), (x2, r2) = out
    assert np.array_equal(x1, x2) and [r.iters for r in r1] == [r.iters for r in r2]
    assert all(r.converged for r in r1)


@pytest.mark.gpu
@pytest.mark.parametrize("i,j", [(31, 10), (5, 31), (31, 31)])
def test_wait_for_another_cluster_runs_out(i, j):
    """A column at a cluster's edge never arrives: the polling warp's wait, the waits of the
    cells behind it and of the clusters after it end, and the next solve is as before."""
    m = box_mesh(35, 37, 6)
    c = _context(m)
    a, su = c.laplacian(*poisson_system(m))
    x0 = np.zeros(m.numCells)
    before = {s: getattr(c, s)(a, su, x0, 0.0, 6).fi for s in ("iccg", "bicgstab")}
    c.set_sweep_wait_test(polls=4096, absent_row=1 + i + 35 * (j + 37 * 2))
    for solver in before:
        with pytest.raises(_lib.FcgError) as ei:
            getattr(c, solver)(a, su, x0, 0.0, 6)
        assert ei.value.status == _lib.FCG_ERR_TIMEOUT and "dependency wait" in str(ei.value)
    c.set_sweep_wait_test(0, 0)
    for solver, fi in before.items():
        assert np.array_equal(getattr(c, solver)(a, su, x0, 0.0, 6).fi, fi)
    c.close()
