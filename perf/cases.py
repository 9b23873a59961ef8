"""The work that a user of this package has it do, as cases that can be timed and checked.

A case is one call, or the few calls that always go together, of a flow solver's outer
iteration: gradients, momentum assembly, pressure assembly, the pressure solves, the
transport solves, the batched solves and the learned preconditioner's solve and training
gradient.  Meshes are hexahedral boxes with jittered vertices (numbered as a lexicographic
block) and the same with a step cut out of the inlet corner (numbered as a general
unstructured mesh).  The mesh, its bound context and the network's handle are what a
program keeps over its time steps, so they are kept from one preparation to the next;
everything else is made from the seed.
"""
import gc
import math

import numpy as np
import torch

import freecappuccino_gb300 as fcg
from freecappuccino_gb300.learned import DEFAULT_WEIGHTS, LearnedPreconditioner
from freecappuccino_gb300.systems import transport_systems

DEV = "cuda"
F64 = torch.float64
SMALL = float(np.float32(1e-20))


def listed():
    return [
        # a tutorial-size case driven from host arrays, as the Fortran drivers call it:
        # assembly and a sweep-limited solve, bound by launches and copies
        dict(name="tutorial_host_24", kind="solve", solver="dpcg", nx=24, ny=24, nz=24, step=False,
             sweeps=30, host=True),
        # the gradients of u, v, w and p that open every outer iteration
        dict(name="gradients_128", kind="gradients", method="gauss", passes=1, nx=128, ny=128,
             nz=128, step=False),
        # the momentum equations' assembly with the default face-value scheme
        dict(name="momentum_96", kind="momentum", scheme="muscl", nx=96, ny=96, nz=96, step=False),
        # the pressure-correction assembly with Rhie-Chow fluxes, and the flux, field and
        # non-orthogonal corrections that follow its solve
        dict(name="pressure_assembly_128", kind="pressure", nx=128, ny=128, nz=128, step=False),
        # the reference's own pressure solver, stopped at its sweep limit as inside an
        # outer iteration, on a block ...
        dict(name="iccg_128", kind="solve", solver="iccg", nx=128, ny=128, nz=128, step=False,
             sweeps=40, host=False),
        # ... and on a mesh that is not one, with odd extents
        dict(name="iccg_step_93x81x77", kind="solve", solver="iccg", nx=93, ny=81, nz=77, step=True,
             sweeps=40, host=False),
        # the five transport systems of a time step (u, v, w, k, epsilon) in one call
        dict(name="transport_5x128", kind="transport", nsys=5, nx=128, ny=128, nz=128, step=False),
        # independent pressure solves of uneven sizes in one launch
        dict(name="batch_12", kind="batch", sizes="32,48,64,96,128,32,96,64,48,128,64,96",
             sweeps=150),
        # one pass of the network on a mesh that is not a block
        dict(name="network_step_97", kind="network", nx=97, ny=90, nz=85, step=True),
        # a training gradient: forward and backward of one (residual, error) pair
        dict(name="train_64", kind="train", nx=64, ny=64, nz=64, step=False),
        # whole solves by the flexible CG, to a tight tolerance as a time-accurate step takes
        # them: Jacobi sweeps with the coarse-grid correction on an ordinary mesh ...
        dict(name="fcg_jacobi_160", kind="fcg", smoother="jacobi", ml_sweeps=2, nx=160, ny=160,
             nz=160, step=False),
        # ... and the learned preconditioner on the largest one
        dict(name="fcg_network_256", kind="fcg", smoother="network", ml_sweeps=3, nx=256, ny=256,
             nz=256, step=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _extents(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return dict(nx=n, ny=max(lo, int(n * rng.uniform(0.7, 1.0))),
                nz=max(lo, int(n * rng.uniform(0.7, 1.0))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "gradients", "momentum", "pressure", "transport",
                       "batch", "network", "train", "fcg", "fcg"])
    step = rng.random() < 0.35
    if kind == "solve":
        host = rng.random() < 0.2
        solver = rng.choice(["dpcg", "iccg", "iccg", "bicgstab", "dpcg_mixed"])
        return dict(kind=kind, solver=solver, step=step, host=host,
                    sweeps=2000 if solver == "dpcg_mixed" else rng.randint(10, 60),
                    **_extents(rng, 16, 48 if host else 144))
    if kind == "gradients":
        method = rng.choice(["gauss", "gauss", "lsq"])
        return dict(kind=kind, method=method, passes=rng.choice([1, 2]) if method == "gauss" else 1,
                    step=step, **_extents(rng, 16, 140))
    if kind == "momentum":
        return dict(kind=kind, scheme=rng.choice(["muscl", "central", "second_upwind", "cds"]),
                    step=step, **_extents(rng, 16, 110))
    if kind == "pressure":
        return dict(kind=kind, step=step, **_extents(rng, 16, 140))
    if kind == "transport":
        return dict(kind=kind, nsys=rng.choice([1, 3, 5]), step=step, **_extents(rng, 24, 120))
    if kind == "batch":
        return dict(kind=kind, sizes=",".join(str(_log_int(rng, 20, 110))
                                              for _ in range(rng.randint(4, 14))),
                    sweeps=rng.randint(20, 150))
    if kind == "network":
        return dict(kind=kind, step=step, **_extents(rng, 24, 130))
    if kind == "train":
        return dict(kind=kind, step=False, **_extents(rng, 24, 90))
    return dict(kind=kind, smoother=rng.choice(["network", "jacobi"]), ml_sweeps=rng.choice([2, 3]),
                step=step, **_extents(rng, 32, 150))


# ---------------------------------------------------------------------------------------
# meshes and what a program keeps with them
# ---------------------------------------------------------------------------------------
_kept = {}


def _box_mesh(nx, ny, nz, step):
    """nx x ny x nz cells of the jittered hex mesh; with `step`, without the cells of the
    inlet corner (a backward-facing step).  Returns the mesh and i + j + k of its cells."""
    N = max(nx, ny, nz)
    cube = nx == ny == nz and not step
    m = fcg.hex_mesh(N, jitter=0.2, seed=7, keep_topology=not cube, device=0)
    c = np.arange(N ** 3)
    i, j, k = c % N, (c // N) % N, c // (N * N)
    if cube:
        return m, i + j + k
    inside = (i < nx) & (j < ny) & (k < nz)
    cut = (i < nx // 4) & (j < ny // 3) if step else np.zeros(N ** 3, bool)
    keep = inside & ~cut
    new = np.cumsum(keep)  # 1-based numbers of the cells that stay
    nin = m.numInnerFaces
    P, Q = m.owner[:nin] - 1, m.neighbour - 1
    kp, kq = keep[P], keep[Q]
    nodes = m.face_nodes.reshape(-1, 4)
    inner = np.flatnonzero(kp & kq)
    one = np.flatnonzero(kp ^ kq)  # a face that becomes a boundary face
    flip = ~kp[one]
    own1 = np.where(flip, Q[one], P[one])
    gone = np.where(flip, P[one], Q[one])
    nod1 = np.where(flip[:, None], nodes[one][:, ::-1], nodes[one])
    parts = {"symmetry": [], "wall": []}
    for typ, cnt, st in (("symmetry", "nsym", "iSymmetryFacesStart"),
                         ("wall", "nwal", "iWallFacesStart")):
        f = np.arange(m.starts[st], m.starts[st] + m.counts[cnt])
        f = f[keep[m.owner[f] - 1]]
        sel = inside[gone] if typ == "wall" else ~inside[gone]
        parts[typ] = [np.concatenate([m.owner[f] - 1, own1[sel]]),
                      np.concatenate([nodes[f], nod1[sel]])]
    ns, nw = len(parts["symmetry"][0]), len(parts["wall"][0])
    owner = new[np.concatenate([P[inner], parts["symmetry"][0], parts["wall"][0]])]
    face_nodes = np.concatenate([nodes[inner], parts["symmetry"][1], parts["wall"][1]])
    out = fcg.polymesh_mesh(m.points, np.arange(len(owner) + 1, dtype=np.int32) * 4,
                            np.ascontiguousarray(face_nodes.reshape(-1)).astype(np.int32),
                            owner.astype(np.int32), new[Q[inner]].astype(np.int32),
                            int(keep.sum()), ["symmetry", "wall"], [ns, nw],
                            [len(inner), len(inner) + ns], device=0)
    out.points = out.face_ptr = out.face_nodes = None
    return out, (i + j + k)[keep]


def _keep(key, make):
    if key not in _kept:
        _kept.clear()
        gc.collect()
        torch.cuda.empty_cache()
        _kept[key] = make()
    return _kept[key]


class _Plan:
    """A mesh, its bound context and its arrays on the device."""

    def __init__(self, nx, ny, nz, step, learned=False, transport=0):
        self.mesh, self.level = _box_mesh(nx, ny, nz, step)
        m = self.mesh
        self.ctx = fcg.Context(m)
        self.n, self.ntot, self.nin = m.numCells, m.numTotal, m.numInnerFaces
        t = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(DEV)  # noqa: E731
        self.xc = torch.stack([t(m.xc), t(m.yc), t(m.zc)], 1)
        self.vol = t(m.vol)
        bf = [np.arange(m.starts[s], m.starts[s] + m.counts.get(c, 0))
              for s, c in (("iSymmetryFacesStart", "nsym"), ("iWallFacesStart", "nwal"))]
        self.bfaces = np.concatenate(bf)  # in the order of the boundary slots
        self.nsym = len(bf[0])
        self.xb = torch.stack([t(a[self.bfaces]) for a in (m.xf, m.yf, m.zf)], 1)
        self.lp = None
        if learned:
            self.lp = LearnedPreconditioner(path=DEFAULT_WEIGHTS)
        if transport:
            a, _, dt = transport_systems(m, self.ctx.create_csr(), seed=1, nsys=transport)
            self.a, self.dt = t(a), dt
            self.diag = t(self.ctx.create_csr()[2].astype(np.int64) - 1)


def _plan(case, **kw):
    key = tuple(case[k] for k in ("nx", "ny", "nz", "step")) + tuple(sorted(kw.items()))
    return _keep(key, lambda: _Plan(*key[:4], **kw))


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape, lo=-1.0, hi=1.0, dtype=F64):
    return torch.rand(*shape, generator=g, device=DEV, dtype=dtype) * (hi - lo) + lo


def _smooth(g, x):
    """A smooth field at the points x, three Fourier modes, and its gradient."""
    k = 2 * math.pi * torch.floor(_rand(g, 3, 3, lo=1.0, hi=4.0))
    ph, am = _rand(g, 3, lo=0.0, hi=6.28), _rand(g, 3, lo=0.2, hi=0.5)
    v, d = torch.zeros(len(x), dtype=F64, device=DEV), torch.zeros_like(x)
    for j in range(3):
        arg = (x * k[j]).sum(1) + ph[j]
        v += am[j] * torch.sin(arg)
        d += am[j] * torch.cos(arg)[:, None] * k[j]
    return v, d


def _poisson(p, g):
    """A pressure system: smooth diffusivity between about 0.2 and 5, U(-1,1) vol on the right."""
    mu = -torch.exp(_smooth(g, p.xc)[0])
    su = _rand(g, p.n) * p.vol
    phi = torch.zeros(p.ntot, dtype=F64, device=DEV)
    a, su = p.ctx.laplacian(mu, phi, su)
    return mu, phi, a, su


def _flow(p, g):
    """Velocity, pressure, density and momentum coefficients of an outer iteration."""
    x = torch.cat([p.xc, p.xb])
    f = {}
    for k, name in (("u", "dUdxi"), ("v", "dVdxi"), ("w", "dWdxi"), ("p", "dPdxi")):
        v, d = _smooth(g, x)
        f[k] = v + 0.01 * _rand(g, p.ntot)
        f[name] = d[:p.n].contiguous()
    f["den"] = 1.0 + 0.2 * _rand(g, p.ntot)
    for k in ("apu", "apv", "apw"):
        f[k] = (1.0 + 0.1 * _rand(g, p.n)) / p.vol
    return f


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "batch":
        sizes = [int(s) for s in case["sizes"].split(",")]

        def make():
            plans = [_Plan(s, s, s, False) for s in sizes]
            return plans, fcg.Batch([p.ctx for p in plans])

        plans, batch = _keep((kind, case["sizes"]), make)
        sys_ = [_poisson(p, g) for p in plans]
        torch.cuda.synchronize()
        return dict(case=case, batch=batch, plans=plans, a=[s[2] for s in sys_],
                    su=[s[3] for s in sys_],
                    fi=[torch.zeros(p.n, dtype=F64, device=DEV) for p in plans])
    if kind == "transport":
        p = _plan(case, transport=case["nsys"])
        a = p.a.clone()
        a[:, p.diag] += 0.2 * _rand(g, 1, lo=0.0) * p.vol / p.dt  # another time step
        return dict(case=case, p=p, a=a, su=_rand(g, case["nsys"], p.n) * p.vol,
                    fi=torch.zeros(case["nsys"], p.n, dtype=F64, device=DEV))
    if kind in ("network", "train", "fcg"):
        p = _plan(case, learned=True)
        _, _, a, su = _poisson(p, g)
        s = dict(case=case, p=p, a=a, su=su)
        if kind == "fcg":
            s["fi"] = torch.zeros(p.n, dtype=F64, device=DEV)
            p.lp.set_multilevel(smoother=case["smoother"], sweeps=case["ml_sweeps"])
            return s
        # a residual and its error in the scaled system, as the solver's iterates have them
        x = _smooth(g, p.xc)[0] + 0.1 * _rand(g, p.n)
        r = p.ctx.spmv(a, x)
        dg = torch.from_numpy(p.ctx.create_csr()[2].astype(np.int64) - 1).to(DEV)
        d = a[dg].sqrt()
        s["r"], s["e"] = (r / d).float(), (x * d).float()
        return s
    p = _plan(case)
    if kind == "solve":
        mu, phi, a, su = _poisson(p, g)
        s = dict(case=case, p=p, mu=mu, phi=phi, a=a, su=su,
                 su0=torch.zeros(p.n, dtype=F64, device=DEV),
                 fi=torch.zeros(p.n, dtype=F64, device=DEV))
        if case["host"]:
            s["su0"] = _rand(g, p.n) * p.vol
            for k in ("mu", "phi", "su0", "fi"):
                s[k] = s[k].cpu().numpy()
        return s
    f = _flow(p, g)
    s = dict(case=case, p=p, f=f)
    if kind == "momentum":
        f["vis"] = 1e-3 * (1.0 + 0.5 * _rand(g, p.ntot, lo=0.0))
        f["flmass"] = 0.05 * _rand(g, p.nin) * p.vol.mean() ** (2.0 / 3.0)
        f["den"] = f["den"][:p.n].contiguous()
        s["a"] = _rand(g, p.n + 2 * p.nin)
    if kind == "pressure":
        s["pp"] = _smooth(g, torch.cat([p.xc, p.xb]))[0]
        s["dpp"] = _smooth(g, p.xc)[1]
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "batch":
        return s["batch"].dpcg(s["a"], s["su"], s["fi"], 1e-8, c["sweeps"])[0]
    p = s["p"]
    if kind == "gradients":
        f = s["f"]
        if c["method"] == "lsq":
            return [p.ctx.grad(f[k], "lsq") for k in "uvwp"]
        return [p.ctx.grad(f[k], "gauss", c["passes"]) for k in "uvwp"]
    if kind == "momentum":
        f = s["f"]
        return p.ctx.calcuvw(f["u"], f["v"], f["w"], f["p"], f["vis"], f["den"], f["dUdxi"],
                             f["dVdxi"], f["dWdxi"], f["dPdxi"], f["flmass"], s["a"],
                             scheme=c["scheme"])
    if kind == "pressure":
        f = s["f"]
        a, su, fm = p.ctx.facefluxmass(*[f[k] for k in (
            "u", "v", "w", "p", "dUdxi", "dVdxi", "dWdxi", "dPdxi", "apu", "apv", "apw", "den")])
        fm = p.ctx.flux_correct(a, s["pp"], fm)
        u, v, w, q = p.ctx.correct_fields(s["dpp"], f["apu"], f["apv"], f["apw"], s["pp"], 0.3, 1,
                                          f["u"], f["v"], f["w"], f["p"])
        su2, fm = p.ctx.fluxmc(s["dpp"], f["apu"], f["den"], fm)
        return [a, su, fm, u, v, w, q, su2]
    if kind == "transport":
        return p.ctx.bicgstab_multi(s["a"], s["su"], s["fi"], 1e-10, 200)[0]
    if kind == "network":
        p.lp.set_matrix(p.ctx, s["a"])
        return p.lp.apply(p.ctx, s["r"])
    if kind == "train":
        p.lp.set_matrix(p.ctx, s["a"])
        return p.lp.loss_grad(p.ctx, s["r"], s["e"])
    if kind == "fcg":
        return p.lp.solve(p.ctx, s["a"], s["su"], s["fi"], 1e-11, 2000).fi
    a, su = s["a"], s["su"]
    if c["host"]:
        a, su = p.ctx.laplacian(s["mu"], s["phi"], s["su0"])
    if c["solver"] == "dpcg_mixed":
        return p.ctx.dpcg_mixed(a, su, s["fi"], 1e-11, c["sweeps"]).fi
    r = getattr(p.ctx, c["solver"])(a, su, s["fi"], 1e-8, c["sweeps"])
    return [r.fi, r.res]


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = sum(int(s) ** 3 for s in case["sizes"].split(","))
        return {"bytes": n * (case["sweeps"] * (56 + 48) + 80), "flops": case["sweeps"] * 24 * n}
    n = case["nx"] * case["ny"] * case["nz"]
    if case["step"]:
        n -= (case["nx"] // 4) * (case["ny"] // 3) * case["nz"]
    if kind == "gradients":  # field in and gradient out; face areas, weights, volumes once
        return {"bytes": 4 * n * 32 + n * (3 * 32 + 8), "flops": 4 * n * 3 * 12}
    if kind == "momentum":   # fields, gradients, face geometry, old matrix; systems out
        return {"bytes": n * (5 * 8 + 4 * 24 + 3 * 8 * 9 + 56 + 56 + 16 + 48), "flops": 3 * n * 220}
    if kind == "pressure":
        return {"bytes": n * (8 * 8 + 5 * 24 + 3 * 8 * 8 + 56 + 24 + 6 * 8), "flops": 3 * n * 150}
    if kind == "transport":  # about 16 products with FP32 copies of the five systems
        return {"bytes": case["nsys"] * n * (56 * 3 + 16 * (28 + 24)), "flops": case["nsys"] * n * 400}
    if kind == "network":    # six layers: the matrix, the features, the residual in, z out
        return {"bytes": n * (28 + 24 + 4 + 4), "flops": 6 * n * (4096 + 448)}
    if kind == "train":
        return {"bytes": n * (28 + 24 + 8) * 3, "flops": 3 * 6 * n * (4096 + 448)}
    if kind == "fcg":        # about 40 iterations, each a fine product and a cycle
        net = 6 * (4096 + 448) if case["smoother"] == "network" else 0
        return {"bytes": n * 40 * (28 * 2 + 40), "flops": n * 40 * (net + 60)}
    if case["solver"] == "dpcg_mixed":  # about 5 sweeps per cell of the longest edge
        return {"bytes": n * 5 * max(case["nx"], 16) * (28 + 24), "flops": n * 5 * case["nx"] * 24}
    per = {"dpcg": 104, "iccg": 220, "bicgstab": 400}[case["solver"]]
    return {"bytes": n * (case["sweeps"] * per + 80), "flops": n * case["sweeps"] * per // 4}


# ---------------------------------------------------------------------------------------
# the same results in 64 bits from plain torch
# ---------------------------------------------------------------------------------------
class _Sparse:
    """A matrix on a mesh's pattern, CSR with ascending columns, from its face list."""

    def __init__(self, p, a=None):
        m, n = p.mesh, p.n
        P = torch.from_numpy(m.owner[:p.nin].astype(np.int64) - 1).to(DEV)
        Q = torch.from_numpy(m.neighbour.astype(np.int64) - 1).to(DEV)
        i = torch.arange(n, device=DEV)
        key = torch.cat([i * n + i, P * n + Q, Q * n + P])
        key = torch.sort(key)[0]
        self.n, self.row, self.col = n, key // n, key % n
        del key
        self.ptr = torch.searchsorted(self.row, torch.arange(n + 1, device=DEV))
        self.isd = self.row == self.col
        if a is not None:
            self.set(a)

    def set(self, a):
        self.val = a
        self.d = a[self.isd]
        self.A = torch.sparse_csr_tensor(self.ptr, self.col, a, (self.n, self.n))
        return self

    def __matmul__(self, x):
        return self.A @ x

    def cg(self, b, tol):
        x, r = torch.zeros_like(b), b.clone()
        p = z = r / self.d
        rz, b0 = r @ z, r.norm()
        for it in range(6000):
            q = self.A @ p
            al = rz / (p @ q)
            x = x + al * p
            r = r - al * q
            if it % 16 == 0 and r.norm() < tol * b0:
                break
            z = r / self.d
            rz, old = r @ z, rz
            p = z + (rz / old) * p
        return x

    def krylov(self, b, sweeps, precond=None):
        """`sweeps` steps of preconditioned CG from zero: (x, residual)."""
        x, r = torch.zeros_like(b), b.clone()
        p, old = torch.zeros_like(b), 1e20
        res0 = r.abs().sum()
        for _ in range(sweeps):
            z = precond(r) if precond else r / self.d
            rz = r @ z
            p = z + (rz / old) * p
            q = self.A @ p
            al = rz / (p @ q)
            x, r, old = x + al * p, r - al * q, rz
            if r.abs().sum() / (res0 + SMALL) < 1e-8:
                break
        return x, r

    def dic(self, level):
        """The diagonal incomplete Cholesky preconditioner, level by level."""
        lev = torch.from_numpy(level).to(DEV)
        order = torch.argsort(lev, stable=True)
        cnt = torch.bincount(lev).tolist()
        sides = []
        for sel in (self.col < self.row, self.col > self.row):
            e = torch.nonzero(sel)[:, 0]
            rank = torch.zeros_like(e)
            r = self.row[e]
            for k in (1, 2):
                rank[k:] += (r[k:] == r[:-k]).long()
            idx = torch.full((self.n, 3), self.n, device=DEV)
            val = torch.zeros(self.n, 3, dtype=F64, device=DEV)
            idx[r, rank], val[r, rank] = self.col[e], self.val[e]
            sides.append((idx[order], val[order]))
        steps, at = [], 0
        for k in cnt:
            if k:
                steps.append((order[at:at + k], *[x[at:at + k] for s in sides for x in s]))
            at += k
        D = torch.zeros(self.n + 1, dtype=F64, device=DEV)
        for c, li, lv, _, _ in steps:
            D[c] = 1.0 / (self.d[c] - (lv * lv * D[li]).sum(1))

        def apply(r):
            z = torch.zeros(self.n + 1, dtype=F64, device=DEV)
            for c, li, lv, _, _ in steps:
                z[c] = (r[c] - (lv * z[li]).sum(1)) * D[c]
            y = z[:self.n] / (D[:self.n] + SMALL)
            z.zero_()
            for c, _, _, ui, uv in reversed(steps):
                z[c] = (y[c] - (uv * z[ui]).sum(1)) * D[c]
            return z[:self.n]

        return apply


class _Faces:
    """Inner-face geometry of a mesh as torch arrays."""

    def __init__(self, p):
        m, nin = p.mesh, p.nin
        t = lambda *a: torch.stack([torch.from_numpy(np.ascontiguousarray(x)) for x in a], 1).to(DEV)  # noqa: E731
        self.P = torch.from_numpy(m.owner[:nin].astype(np.int64) - 1).to(DEV)
        self.N = torch.from_numpy(m.neighbour.astype(np.int64) - 1).to(DEV)
        S, xf = t(m.arx, m.ary, m.arz), t(m.xf, m.yf, m.zf)
        self.S, self.xf = S[:nin], xf[:nin]
        self.Sb, self.xb = S[p.bfaces], xf[p.bfaces]
        self.own = torch.from_numpy(m.owner[p.bfaces].astype(np.int64) - 1).to(DEV)
        self.lam = torch.from_numpy(m.facint).to(DEV)
        self.n, self.nsym, self.xc, self.vol = p.n, p.nsym, p.xc, p.vol
        self.are = self.S.norm(dim=1)
        self.d = self.xc[self.N] - self.xc[self.P]

    def mean(self, x):
        w = self.lam if x.dim() == 1 else self.lam[:, None]
        return x[self.P] * (1 - w) + x[self.N] * w

    def div(self, fP, fN=None):
        """Per cell, the face terms added as owner and (default: minus them) as neighbour."""
        out = torch.zeros((self.n,) + fP.shape[1:], dtype=F64, device=DEV)
        return out.index_add_(0, self.P, fP).index_add_(0, self.N, -fP if fN is None else fN)

    def central(self, fi, g):
        """face_value_central: the mean of both cells' linear extrapolations."""
        c = (g[self.P] * (self.xf - self.xc[self.P])).sum(1) + \
            (g[self.N] * (self.xf - self.xc[self.N])).sum(1)
        return 0.5 * (fi[self.P] + fi[self.N] + c)

    def matrix(self, pn, np_, diag):
        """CSR values, columns ascending, of the off-diagonals per face and the diagonal."""
        i = torch.arange(self.n, device=DEV)
        key = torch.cat([i * self.n + i, self.P * self.n + self.N, self.N * self.n + self.P])
        return torch.cat([diag, pn, np_])[torch.argsort(key)]


def _exact_gradients(p, f, passes):
    t, out = _Faces(p), []
    for k in "uvwp":
        fi, fb = f[k][:p.n], f[k][p.n:]
        g = torch.zeros(p.n, 3, dtype=F64, device=DEV)
        for _ in range(passes):
            fe = t.mean(fi) + (t.mean(g) * (t.xf - t.mean(p.xc))).sum(1)
            g = t.div(fe[:, None] * t.S).index_add_(0, t.own, fb[:, None] * t.Sb) / p.vol[:, None]
        out.append(g)
    return out


def _exact_pressure(s):
    p, f = s["p"], s["f"]
    t = _Faces(p)
    nrm = t.S / t.are[:, None]
    ap = torch.stack([f["apu"], f["apv"], f["apw"]], 1) * p.vol[:, None]
    D, den = t.mean(ap), t.mean(f["den"][:p.n])
    sfr = 1.0 / (t.S * t.d * nrm).sum(1)
    cap = -den * D[:, 0] * t.are ** 2 * sfr
    uf = torch.stack([t.central(f[k], f[g]) for k, g in
                      (("u", "dUdxi"), ("v", "dVdxi"), ("w", "dWdxi"))], 1)
    off = lambda c: t.xf - (t.xf - c) * nrm - c  # noqa: E731
    xP, xN, dP = off(p.xc[t.P]), off(p.xc[t.N]), f["dPdxi"]
    sign = torch.tensor([-1.0, 1.0, 1.0], dtype=F64, device=DEV)
    dpe = f["p"][t.N] - f["p"][t.P] + (dP[t.N] * xN).sum(1) + (sign * dP[t.P] * xP).sum(1)
    ue = uf - D * (dpe * sfr)[:, None] * t.S + D * t.mean(dP) * t.d * nrm
    fm = den * (ue * t.S).sum(1)
    a = t.matrix(cap, cap, t.div(-cap, -cap))
    su = -t.div(fm)
    pp, dpp = s["pp"], s["dpp"]
    fm = fm + cap * (pp[t.N] - pp[t.P])
    new = [f[k].clone() for k in "uvw"]
    for k, x in enumerate(new):
        x[:p.n] -= dpp[:, k] * ap[:, k]
    q = f["p"].clone()
    q[:p.n] += 0.3 * (pp[:p.n] - pp[0])
    cor = t.mean(f["apu"] * f["den"][:p.n] * p.vol) * t.are / (t.d * nrm).sum(1) * \
        ((dpp[t.N] * xN).sum(1) - (dpp[t.P] * xP).sum(1))
    return [a, su, fm + cor, *new, q, -t.div(cor)]


def _exact_momentum(s, scheme):
    p, f = s["p"], s["f"]
    t = _Faces(p)
    n, fm = p.n, f["flmass"]
    # the pressure divergence reads the (3, n) gradient array as element cell + 3 k
    flat = f["dPdxi"].reshape(-1)
    dp = torch.stack([t.mean(flat[3 * k:3 * k + n]) for k in range(3)], 1)
    pe = t.mean(f["p"][:n]) + (dp * (t.xf - t.mean(p.xc))).sum(1)
    S = -t.div(pe[:, None] * t.S).index_add_(0, t.own, f["p"][n:, None] * t.Sb)
    visc = t.mean(f["vis"][:n])
    de = visc * t.are / t.d.norm(dim=1)
    can, cap = -de + fm.clamp(max=0), -de - fm.clamp(min=0)
    U = [f[k] for k in "uvw"]
    G = [f[k] for k in ("dUdxi", "dVdxi", "dWdxi")]
    gi = [t.mean(g) for g in G]
    r = t.S / (t.d * t.S).sum(1)[:, None]
    gn = torch.stack([gi[c] + r * (U[c][t.N] - U[c][t.P] - (gi[c] * t.d).sum(1))[:, None]
                      for c in range(3)], 1)
    fde = visc[:, None] * ((gn + gn.transpose(1, 2)) * t.S[:, None, :]).sum(2)
    up = fm >= 0
    first = torch.where(up, t.P, t.N)
    for c in range(3):
        fi, g = U[c], G[c]
        upw = fi[first] + (g[first] * (t.xf - p.xc[first])).sum(1)
        fv = {"cds": lambda: fi[t.P] * t.lam + fi[t.N] * (1 - t.lam),  # as the reference weighs it
              "central": lambda: t.central(fi, g), "second_upwind": lambda: upw,
              "muscl": lambda: 0.125 * t.central(fi, g) + 0.875 * upw}[scheme]()
        src = -(fm * (fv - fi[first])) + fde[:, c] - de * (gi[c] * t.d).sum(1)
        S[:, c] += t.div(src)
    SP = torch.zeros(n, 3, dtype=F64, device=DEV)
    nb, own, ns = t.Sb / t.Sb.norm(dim=1, keepdim=True), t.own, t.nsym
    dn = ((t.xb - p.xc[own]) * nb).sum(1)
    V = torch.stack([u[:n][own] - u[n:] for u in U], 1)
    vis = torch.cat([f["vis"][n:n + ns], torch.full_like(f["vis"][n + ns:], 1e-3)])
    are = t.Sb.norm(dim=1)
    cf, vs = vis * are / dn, vis * are / (t.xb - p.xc[own]).norm(dim=1)
    vn = (V * nb).sum(1)
    fd = torch.cat([2 * cf[:ns, None] * vn[:ns, None] * nb[:ns],
                    cf[ns:, None] * (V - vn[:, None] * nb)[ns:]])
    SP.index_add_(0, own, vs[:, None].expand(-1, 3).contiguous())
    uc = torch.stack([u[:n] for u in U], 1)
    S.index_add_(0, own, vs[:, None] * uc[own] - fd)
    dg = (SP - t.div(can, cap)[:, None]) / 0.7
    rhs = S + 0.3 * dg * uc
    return dict(a=t.matrix(can, cap, dg[:, 0]), diag_vw=dg[:, 1:].T.contiguous(),
                rhs=rhs.T.contiguous(), ap=(1.0 / dg).T.contiguous())


def _network(p, a, r, e, w):
    """The network (and, with e, its loss and gradient) in 64 bits."""
    A = _Sparse(p, a)
    s = 1.0 / A.d.sqrt()
    A.set(a * s[A.row] * s[A.col])
    t = _Faces(p)
    h3 = p.vol ** (1.0 / 3.0)
    areas = t.div(t.S.abs(), t.S.abs()).index_add_(0, t.own, t.Sb.abs()) / (2 * h3 * h3)[:, None]
    r = r.double()
    rms = (r @ r / p.n).sqrt()
    d = 1.0 / (s * s)
    x = torch.cat([(r / rms)[:, None], torch.log(d / h3 / 6.0)[:, None],
                   torch.log(p.vol / p.vol.mean())[:, None], areas - 1.0], 1)

    class Mul(torch.autograd.Function):  # the matrix is symmetric
        @staticmethod
        def forward(ctx, h):
            return A.A @ h

        @staticmethod
        def backward(ctx, g):
            return A.A @ g.contiguous()

    w = torch.from_numpy(w).to(DEV, F64).requires_grad_(e is not None)
    at = [0]

    def take(*shape):
        k = math.prod(shape)
        at[0] += k
        return w[at[0] - k:at[0]].reshape(shape)

    W, b = take(32, 6), take(32)
    h = torch.relu(x @ W.T + b)
    for _ in range(6):
        W, b = take(32, 64), take(32)
        h = h + torch.relu(torch.cat([h, Mul.apply(h)], 1) @ W.T + b)
    y = x[:, 0] + h @ take(32) + take(1)
    if e is None:
        return rms * y
    T = A.A @ (e.double() / rms)[:, None]
    R = Mul.apply(y[:, None]) - T
    loss = (R * R).sum() / (T * T).sum()
    return loss.item(), torch.autograd.grad(loss, w)[0].cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "batch":
        return [_Sparse(p, a).krylov(su, case["sweeps"])[0]
                for p, a, su in zip(s["plans"], s["a"], s["su"])]
    p = s["p"]
    if kind == "gradients":
        # the reference's least-squares solve swaps signs in one row: no plain value
        return None if case["method"] == "lsq" else \
            _exact_gradients(p, s["f"], case["passes"])
    if kind == "momentum":
        return _exact_momentum(s, case["scheme"])
    if kind == "pressure":
        return _exact_pressure(s)
    if kind == "transport":
        A, out = _Sparse(p), []
        for k in range(case["nsys"]):
            A.set(s["a"][k].contiguous())
            b, x = s["su"][k], s["su"][k] / A.d
            for it in range(400):  # diagonally dominant: Jacobi converges fast
                r = b - A @ x
                x = x + r / A.d
                if it % 8 == 0 and r.norm() < 1e-14 * b.norm():
                    break
            out.append(x)
        return torch.stack(out)
    if kind == "network":
        return _network(p, s["a"], s["r"], None, p.lp.weights)
    if kind == "train":
        return _network(p, s["a"], s["r"], s["e"], p.lp.weights)
    if kind == "fcg":
        return _Sparse(p, s["a"]).cg(s["su"], 1e-13)
    a, su = s["a"], s["su"]
    if case["host"]:
        su = torch.from_numpy(s["su0"]).to(DEV)  # the walls hold zero
    A = _Sparse(p, a)
    if case["solver"] == "dpcg_mixed":
        return A.cg(su, 1e-13)
    if case["solver"] == "bicgstab":
        return None
    x, r = A.krylov(su, case["sweeps"], A.dic(p.level) if case["solver"] == "iccg" else None)
    return [x.cpu().numpy(), r.cpu().numpy()] if case["host"] else [x, r]
