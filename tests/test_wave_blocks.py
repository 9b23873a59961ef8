"""The wavefront-tiled DIC / DILU sweeps on blocks of unequal extents against the
level-ordered form: tiles and clusters cut at the block's edge, blocks of fewer planes than
a tile has steps, and more planes than one launch takes.  And the level-ordered form on a
mesh whose rows hold more entries of one triangle than it keeps in registers.  All forms
use the same row arithmetic in the same entry order, so the same bits."""
import os

import numpy as np
import pytest

import freecappuccino_gb300 as fcg
from tests.meshes import poisson_system

pytestmark = pytest.mark.gpu


def box_mesh(nx, ny, nz, seed=5):
    """An nx x ny x nz block of the unit cube, vertices inside it jittered, cells and faces
    numbered as hex_mesh numbers them; wall at x = 0, symmetry elsewhere."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1),
                             indexing="ij")[::-1], -1).astype(float)
    inner = np.zeros(g.shape[:3], bool)
    inner[1:-1, 1:-1, 1:-1] = True
    g[inner] += 0.2 * rng.uniform(-1, 1, (inner.sum(), 3))
    pts = (g / [nx, ny, nz]).reshape(-1, 3)
    pid = np.arange(len(pts)).reshape(nz + 1, ny + 1, nx + 1) + 1
    cell = np.arange(nx * ny * nz).reshape(nz, ny, nx) + 1
    quad = {  # the four vertices of the faces at i, j or k, the normal pointing up
        "i": np.stack([pid[:-1, :-1], pid[:-1, 1:], pid[1:, 1:], pid[1:, :-1]], -1),
        "j": np.stack([pid[:-1, :, :-1], pid[1:, :, :-1], pid[1:, :, 1:], pid[:-1, :, 1:]], -1),
        "k": np.stack([pid[:, :-1, :-1], pid[:, :-1, 1:], pid[:, 1:, 1:], pid[:, 1:, :-1]], -1)}
    own, nb, nod = [], [], []
    for q, o, n in ((quad["i"][:, :, 1:-1], cell[:, :, :-1], cell[:, :, 1:]),
                    (quad["j"][:, 1:-1], cell[:, :-1], cell[:, 1:]),
                    (quad["k"][1:-1], cell[:-1], cell[1:])):
        own.append(o.ravel())
        nb.append(n.ravel())
        nod.append(q.reshape(-1, 4))
    own, nb, nod = map(np.concatenate, (own, nb, nod))
    order = np.lexsort((nb, own))
    flip = lambda q: q.reshape(-1, 4)[:, ::-1]  # noqa: E731
    bnd = [(quad["i"][:, :, -1].reshape(-1, 4), cell[:, :, -1]), (flip(quad["j"][:, 0]), cell[:, 0]),
           (quad["j"][:, -1].reshape(-1, 4), cell[:, -1]), (flip(quad["k"][0]), cell[0]),
           (quad["k"][-1].reshape(-1, 4), cell[-1]), (flip(quad["i"][:, :, 0]), cell[:, :, 0])]
    nsym = sum(c.size for _, c in bnd[:5])
    owner = np.concatenate([own[order]] + [c.ravel() for _, c in bnd]).astype(np.int32)
    nodes = np.concatenate([nod[order]] + [q for q, _ in bnd])
    return fcg.polymesh_mesh(pts, 4 * np.arange(len(owner) + 1, dtype=np.int32),
                             np.ascontiguousarray(nodes.ravel(), dtype=np.int32), owner,
                             nb[order].astype(np.int32), nx * ny * nz, ["symmetry", "wall"],
                             [nsym, ny * nz], [len(order), len(order) + nsym])


def _context(m, mode=None):
    saved = os.environ.pop("FCG_SWEEP", None)
    if mode:
        os.environ["FCG_SWEEP"] = mode
    try:
        c = fcg.Context(m)
        c.set_solver_options(float(np.float32(1e-20)), True)  # creates the solver state
    finally:
        os.environ.pop("FCG_SWEEP", None)
        if saved is not None:
            os.environ["FCG_SWEEP"] = saved
    return c


@pytest.mark.parametrize("dims", [(2, 2, 2), (16, 8, 3), (17, 9, 4), (35, 37, 6), (3, 70, 9),
                                  (70, 3, 40), (5, 9, 512), (4, 3, 513), (19, 11, 1030)])
def test_tiled_sweeps_equal_row_sweeps(dims):
    m = box_mesh(*dims)
    assert abs(m.vol.sum() - 1.0) < 1e-12 and m.vol.min() > 0
    ctxs = [_context(m), _context(m, "rows")]
    mu, phi, su0 = poisson_system(m)
    a, su = ctxs[0].laplacian(mu, phi, su0)
    x0 = np.zeros(m.numCells)
    for solver in ("iccg", "bicgstab"):
        for _ in range(2):  # the second solve finds the sentinels as the first left them
            r, o = [getattr(c, solver)(a, su, x0, 0.0, 6) for c in ctxs]
            assert np.array_equal(r.fi, o.fi) and r.resl == o.resl, (dims, solver)
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("dims,nsys", [((17, 9, 4), 1), ((35, 37, 6), 5), ((5, 9, 513), 3)])
def test_tiled_multi_rhs_sweeps_equal_row_sweeps(dims, nsys):
    """The FP32 form, several systems in one launch."""
    from freecappuccino_gb300.systems import transport_systems

    m = box_mesh(*dims)
    out = []
    for mode in (None, "rows"):
        c = _context(m)
        a, su, _ = transport_systems(m, c.create_csr(), nsys=nsys)
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


@pytest.mark.parametrize("N", [3, 11])
def test_level_order_of_a_scattered_numbering(N):
    """Cells numbered at random: up to six entries in a row's triangle, uneven levels."""
    m = fcg.hex_mesh(N, 0.2, seed=3)
    p = np.random.default_rng(N).permutation(m.numCells)
    inv = np.argsort(p)
    m.owner = (p[m.owner - 1] + 1).astype(np.int32)
    m.neighbour = (p[m.neighbour - 1] + 1).astype(np.int32)
    for k in ("xc", "yc", "zc", "vol"):
        setattr(m, k, np.ascontiguousarray(getattr(m, k)[inv]))
    ctxs = [_context(m), _context(m, "levels")]
    mu, phi, su0 = poisson_system(m)
    a, su = ctxs[0].laplacian(mu, phi, su0)
    for solver in ("iccg", "bicgstab"):
        for _ in range(2):
            r, o = [getattr(c, solver)(a, su, np.zeros(m.numCells), 0.0, 5) for c in ctxs]
            assert np.array_equal(r.fi, o.fi) and r.resl == o.resl, (N, solver)
    for c in ctxs:
        c.close()
