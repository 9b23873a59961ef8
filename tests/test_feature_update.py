"""A set_matrix that fails half way leaves nothing behind: the next one, on whatever mesh,
gives what a fresh handle gives."""
import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from freecappuccino_gb300 import _lib
from freecappuccino_gb300.learned import LearnedPreconditioner
from tests.meshes import poisson_system
from tests.test_wave_blocks import box_mesh

pytestmark = pytest.mark.gpu


def _scattered(m, seed):
    """m with its cells numbered at random: no block."""
    p = np.random.default_rng(seed).permutation(m.numCells)
    inv = np.argsort(p)
    m.owner = (p[m.owner - 1] + 1).astype(np.int32)
    m.neighbour = (p[m.neighbour - 1] + 1).astype(np.int32)
    for k in ("xc", "yc", "zc", "vol"):
        setattr(m, k, np.ascontiguousarray(getattr(m, k)[inv]))
    return m


def _handle():
    lp = LearnedPreconditioner(seed=1)
    w = lp.weights  # the output layer starts at zero
    w[-33:-1] = np.linspace(-0.2, 0.2, 32)
    lp.weights = w
    return lp


@pytest.mark.parametrize("block", [False, True])
@pytest.mark.parametrize("other", [(9, 8, 9), (13, 12, 11)])
def test_failed_update_does_not_reach_the_next_mesh(block, other):
    """Fewer cells: the buffers stay, only their owner changes. More cells: they grow. A block
    before and after it also has its stencil values replaced."""
    ma = box_mesh(9, 8, 10) if block else _scattered(box_mesh(9, 8, 10), 3)
    mb = box_mesh(*other)
    ca, cb = fcg.Context(ma), fcg.Context(mb)
    aa, _ = ca.laplacian(*poisson_system(ma))
    ab, _ = cb.laplacian(*poisson_system(mb))
    r = fcg.uniform(5, 0, ma.numCells).astype(np.float32)
    fresh = _handle()
    fresh.set_matrix(ca, aa)
    want = fresh.apply(ca, r), fresh.features(ca)
    lp = _handle()
    lp.set_matrix(ca, aa)
    lp.set_prepare_test(1)
    with pytest.raises(_lib.FcgError):
        lp.set_matrix(cb, ab)
    with pytest.raises(_lib.FcgError):
        lp.apply(cb, np.zeros(mb.numCells, np.float32))  # no features of that mesh
    for _ in range(2):
        lp.set_matrix(ca, aa)
        assert np.array_equal(lp.apply(ca, r), want[0])
        assert np.array_equal(lp.features(ca), want[1])
    lp.set_matrix(cb, ab)  # and the mesh that failed
    fresh.set_matrix(cb, ab)
    rb = fcg.uniform(6, 0, mb.numCells).astype(np.float32)
    assert np.array_equal(lp.apply(cb, rb), fresh.apply(cb, rb))
    for h in (lp, fresh):
        h.close()
    ca.close()
    cb.close()
