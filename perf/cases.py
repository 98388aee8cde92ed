"""The solver's work as its users have it done, one case per kind of program.

Every case goes through the public binding (``dgp.Solver``, ``dgp.Ensemble``):
a program keeps a mesh, a law and a solver, puts a state in, advances it and
takes the state (or a gradient) out.  ``prepare`` makes what the program has
in hand, ``run`` is one pass, ``work`` what a pass cannot do without, and
``exact`` the same values in 64 bits from plain torch: a discontinuous
Galerkin step written out over whole arrays (nodal traces per face, index_add
for the lift), without the library's kernels.

Meshes are the jittered grids of the workloads; states are the laws' fields
projected with seeded parameters.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "dg-parallel_b200"))
import dgp  # noqa: E402

LAWS = {"scalar": dgp.LAW_SCALAR, "burgers": dgp.LAW_BURGERS2D, "euler2d": dgp.LAW_EULER2D,
        "euler3d": dgp.LAW_EULER3D, "maxwell3d": dgp.LAW_MAXWELL3D, "maxwell2d": dgp.LAW_MAXWELL2D}
FLUXES = {"upwind": dgp.FLUX_UPWIND, "central": dgp.FLUX_CENTRAL, "godunov": dgp.FLUX_GODUNOV,
          "roe": dgp.FLUX_ROE, "llf": dgp.FLUX_LLF}
FIELDS = {"scalar": dgp.FIELD_GAUSS, "burgers": dgp.FIELD_SINE, "euler2d": dgp.FIELD_VORTEX,
          "euler3d": dgp.FIELD_PULSE3D, "maxwell3d": dgp.FIELD_TM110, "maxwell2d": dgp.FIELD_TM2D}
NFIELDS = {"scalar": 1, "burgers": 1, "euler2d": 4, "euler3d": 5, "maxwell3d": 6, "maxwell2d": 3}
CFL = 0.1
GAMMA = 1.4


def listed():
    return [
        # the smallest call of a time loop: scalar advection on 2048 triangles,
        # a short stretch of steps between two outputs (launch latency)
        {"name": "advection_p2_2k", "do": "run", "law": "scalar", "flux": "upwind", "dim": 2, "order": 2,
         "nx": 32, "ny": 32, "mixed": False, "workload_rule": False, "steps": 20},
        # the drop-in TimeIntegrator: a host program that owns the state hands
        # it over, has one step taken and takes it back
        {"name": "integrator_step_p2_3k", "do": "step", "law": "euler2d", "flux": "roe", "dim": 2, "order": 2,
         "nx": 45, "ny": 31, "mixed": False, "workload_rule": False, "steps": 1},
        # low order, odd sizes: linear elements with the Lax-Friedrichs flux
        {"name": "euler_p1_llf_18k", "do": "run", "law": "euler2d", "flux": "llf", "dim": 2, "order": 1,
         "nx": 67, "ny": 131, "mixed": False, "workload_rule": False, "steps": 24},
        # the isentropic vortex at its full size, plain and mixed form
        {"name": "vortex_p3_131k", "do": "run", "law": "euler2d", "flux": "roe", "dim": 2, "order": 3,
         "nx": 256, "ny": 256, "mixed": False, "workload_rule": False, "steps": 16},
        {"name": "vortex_p3_131k_mixed", "do": "run", "law": "euler2d", "flux": "roe", "dim": 2, "order": 3,
         "nx": 256, "ny": 256, "mixed": True, "workload_rule": False, "steps": 16},
        # Euler2d's own flux (the exact Riemann solver) on a mid-size mesh
        {"name": "euler_p2_godunov_20k", "do": "run", "law": "euler2d", "flux": "godunov", "dim": 2, "order": 2,
         "nx": 97, "ny": 101, "mixed": False, "workload_rule": False, "steps": 16},
        # the cavity on tets, plain form with the reference's rules (the
        # largest case) and mixed form with the workload's rules
        {"name": "cavity_p2_tet384k", "do": "run", "law": "maxwell3d", "flux": "upwind", "dim": 3, "order": 2,
         "nx": 40, "ny": 40, "mixed": False, "workload_rule": False, "steps": 4},
        {"name": "cavity_p2_tet197k_mixed", "do": "run", "law": "maxwell3d", "flux": "upwind", "dim": 3, "order": 2,
         "nx": 32, "ny": 32, "mixed": True, "workload_rule": True, "steps": 5},
        # 3D gas dynamics on linear tets
        {"name": "pulse3d_p1_tet48k", "do": "run", "law": "euler3d", "flux": "godunov", "dim": 3, "order": 1,
         "nx": 20, "ny": 20, "mixed": False, "workload_rule": False, "steps": 8},
        # a batch of Burgers problems of uneven size and order with the moment
        # limiter, from the initial field
        {"name": "burgers_batch_16", "do": "ensemble", "law": "burgers", "flux": "central", "dim": 2, "order": 4,
         "nx": 1000, "ny": 20000, "count": 16, "mixed": False, "workload_rule": False, "steps": 10},
        # gradient of a receiver objective: forward steps with checkpoints,
        # recompute and backward
        {"name": "adjoint_p2_33k", "do": "adjoint", "law": "euler2d", "flux": "roe", "dim": 2, "order": 2,
         "nx": 128, "ny": 128, "mixed": False, "workload_rule": False, "steps": 20, "every": 5, "receivers": 64},
        # local time stepping on a mesh graded over four size bins
        {"name": "local_steps_p3_33k", "do": "lts", "law": "euler2d", "flux": "roe", "dim": 2, "order": 3,
         "nx": 128, "ny": 128, "ratio": 1.0196, "mixed": False, "workload_rule": False, "steps": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tri", "tri", "tri", "tri", "tet", "tet", "step", "ensemble", "adjoint", "lts"])
    c = {"do": "run", "dim": 2, "mixed": False, "workload_rule": False}
    if kind in ("tri", "step"):
        law, flux = rng.choice([("scalar", "upwind"), ("euler2d", "roe"), ("euler2d", "roe"), ("euler2d", "llf"),
                                ("euler2d", "godunov"), ("burgers", "central"), ("maxwell2d", "upwind")])
        c.update(law=law, flux=flux, order=rng.choice([1, 2, 2, 3, 3, 4]))
        if kind == "step":
            c.update(do="step", nx=_log_int(rng, 12, 120), ny=_log_int(rng, 12, 120), steps=1)
        else:
            big = 256 if c["order"] < 4 else 180
            c.update(nx=_log_int(rng, 24, big), ny=_log_int(rng, 24, big), steps=rng.randint(3, 20),
                     mixed=rng.random() < 0.3)
    elif kind == "tet":
        law, flux = rng.choice([("maxwell3d", "upwind"), ("maxwell3d", "upwind"), ("euler3d", "godunov"),
                                ("scalar", "upwind")])
        order = rng.choice([1, 2, 2])
        n = _log_int(rng, 6, 34 if law == "maxwell3d" else 22)
        mixed = rng.random() < 0.3
        c.update(law=law, flux=flux, dim=3, order=order, nx=n, ny=n, steps=rng.randint(2, 5), mixed=mixed,
                 workload_rule=law == "maxwell3d" and order == 2 and mixed)
    elif kind == "ensemble":
        c.update(do="ensemble", law="burgers", flux="central", order=4, nx=_log_int(rng, 500, 2000),
                 ny=_log_int(rng, 4000, 20000), count=rng.randint(4, 16), steps=rng.randint(3, 10))
    elif kind == "adjoint":
        law, flux = rng.choice([("euler2d", "roe"), ("euler2d", "llf"), ("scalar", "upwind")])
        steps = rng.randint(6, 20)
        c.update(do="adjoint", law=law, flux=flux, order=rng.choice([1, 2, 3]), nx=_log_int(rng, 24, 110),
                 ny=_log_int(rng, 24, 110), steps=steps, every=rng.choice([0, 3, 5]), receivers=rng.randint(8, 64))
    else:
        n = _log_int(rng, 64, 128)
        c.update(do="lts", law="euler2d", flux="roe", order=rng.choice([2, 3]), nx=n, ny=n,
                 ratio=1.0 + 2.5 / n, steps=rng.randint(1, 2))
    return c


# ---------------------------------------------------------------------------
# meshes, bases and quadrature (numpy)

TRI_MONO = [(i - j, j) for i in range(5) for j in range(i + 1)]
TET_MONO = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (0, 2, 0), (0, 0, 2), (1, 1, 0), (1, 0, 1),
            (0, 1, 1)]


def _box(law):
    return 10.0 if law == "euler2d" else 1.0


def _tri_mesh(nx, ny, box, rng, ratio=None):
    """(vertices, cells, boundary edges) of an nx x ny grid cut into triangles:
    interior vertices jittered by 0.15 of the spacing, or graded lines."""
    i, j = (a.ravel() for a in np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="xy"))
    v = np.zeros((len(i), 3))
    if ratio:
        v[:, 0] = box * (ratio ** i - 1.0) / (ratio ** nx - 1.0)
        v[:, 1] = box * (ratio ** j - 1.0) / (ratio ** ny - 1.0)
    else:
        inside = ((i > 0) & (i < nx) & (j > 0) & (j < ny))[:, None]
        h = np.array([box / nx, box / ny])
        v[:, :2] = np.stack([i, j], axis=1) * h + inside * rng.uniform(-0.15, 0.15, (len(i), 2)) * h
    ci, cj = (a.ravel() for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy"))
    p = cj * (nx + 1) + ci
    cells = np.stack([p, p + 1, p + nx + 2, p, p + nx + 2, p + nx + 1], axis=1).reshape(-1, 3)
    return v, cells, _boundary(cells, 2)


def _tet_mesh(n, box, rng):
    """An n^3 grid of cubes, six tets around each main diagonal, vertices
    jittered by 0.1 of the spacing."""
    k, j, i = (a.ravel() for a in np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij"))
    g = np.stack([i, j, k], axis=1)
    inside = ((g > 0) & (g < n)).all(axis=1)[:, None]
    v = (g + inside * rng.uniform(-0.1, 0.1, g.shape)) * (box / n)
    c0 = ((k * (n + 1) + j) * (n + 1) + i)[(g < n).all(axis=1)]
    step = (1, n + 1, (n + 1) ** 2)
    cells = []
    for a, b, c in ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)):
        s1, s2 = step[a], step[a] + step[b]
        cells.append(np.stack([c0, c0 + s1, c0 + s2, c0 + sum(step)], axis=1))
    cells = np.stack(cells, axis=1).reshape(-1, 4)
    e = v[cells[:, 1:]] - v[cells[:, :1]]
    neg = np.linalg.det(e) < 0
    cells[neg, 1], cells[neg, 2] = cells[neg, 2].copy(), cells[neg, 1].copy()
    return v, cells, _boundary(cells, 3)


def _cell_faces(cells, dim):
    """All (cell, face) vertex sets, sorted vertices, and the order that brings equal ones together."""
    sets = [(0, 1), (1, 2), (2, 0)] if dim == 2 else [(0, 1, 2), (0, 1, 3), (1, 2, 3), (0, 2, 3)]
    f = np.sort(np.concatenate([cells[:, s] for s in sets]), axis=1).astype(np.int64)
    key = f[:, 0]
    for a in range(1, dim):
        key = key * (int(cells.max()) + 1) + f[:, a]
    order = np.argsort(key, kind="stable")
    return f, key, order


def _boundary(cells, dim):
    f, key, order = _cell_faces(cells, dim)
    k = key[order]
    alone = np.ones(len(k), dtype=bool)
    same = k[1:] == k[:-1]
    alone[1:] &= ~same
    alone[:-1] &= ~same
    return f[order[alone]]


def _tri_rule(degree):
    """Symmetric rules on the unit triangle (Dunavant 1985), weights of sum 1."""
    orbits = {1: [(1 / 3, 1 / 3, 1.0)],
              2: [(1 / 6, 1 / 6, 1 / 3)],
              3: [(1 / 3, 1 / 3, -0.5625), (0.2, 0.2, 0.52083333333333333)],
              4: [(0.0915762135097707430, 0.0915762135097707430, 0.109951743655321871),
                  (0.445948490915964890, 0.445948490915964890, 0.223381589678011472)],
              5: [(1 / 3, 1 / 3, 0.225), (0.101286507323456343, 0.101286507323456343, 0.125939180544827140),
                  (0.470142064105115109, 0.470142064105115109, 0.132394152788506192)],
              6: [(0.0630890144915022405, 0.0630890144915022405, 0.0508449063702068257),
                  (0.249286745170910401, 0.249286745170910401, 0.116786275726379410),
                  (0.310352451033784449, 0.0531450498448169315, 0.0828510756183735431)],
              8: [(1 / 3, 1 / 3, 0.144315607677787172),
                  (0.459292588292723181, 0.459292588292723181, 0.0950916342672846332),
                  (0.170569307751760213, 0.170569307751760213, 0.103217370534718245),
                  (0.0505472283170309775, 0.0505472283170309775, 0.0324584976231980793),
                  (0.263112829634638112, 0.00839477740995760342, 0.0272303141744349927)]}[degree]
    pts = {}
    for a, b, w in orbits:
        c = 1.0 - a - b
        for p in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b)):
            pts.setdefault((round(p[0], 12), round(p[1], 12)), (p[0], p[1], w))
    r = np.array(list(pts.values()))
    return r[:, :2], r[:, 2] / r[:, 2].sum()


def _tet_rule(degree):
    """A collapsed Gauss rule on the unit tet (weights of sum 1); degree 2: the symmetric 4-point rule."""
    if degree == 2:
        a, b = (5 - math.sqrt(5)) / 20, (5 + 3 * math.sqrt(5)) / 20
        return np.array([[a, a, a], [b, a, a], [a, b, a], [a, a, b]]), np.full(4, 0.25)
    x, w = np.polynomial.legendre.leggauss(degree // 2 + 2)
    x, w = (x + 1) / 2, w / 2
    u, v, s = (a.ravel() for a in np.meshgrid(x, x, x, indexing="ij"))
    wu, wv, ws = (a.ravel() for a in np.meshgrid(w, w, w, indexing="ij"))
    pts = np.stack([u, v * (1 - u), s * (1 - u) * (1 - v)], axis=1)
    wt = wu * wv * ws * (1 - u) ** 2 * (1 - v)
    return pts, wt / wt.sum()


class _Basis:
    """Orthonormal modes of the unit simplex: Gram-Schmidt of the monomials."""

    def __init__(self, dim, order):
        self.mono = [m for m in (TRI_MONO if dim == 2 else TET_MONO) if sum(m) <= order]
        n, f = len(self.mono), math.factorial
        gram = np.array([[math.prod(f(a + b) for a, b in zip(p, q)) / f(sum(p) + sum(q) + dim) for q in self.mono]
                         for p in self.mono], dtype=np.longdouble)
        g = np.zeros((n, n), dtype=np.longdouble)
        for i in range(n):
            v = np.zeros(n, dtype=np.longdouble)
            v[i] = 1
            for _ in range(2):
                for j in range(i):
                    v = v - (v @ gram @ g[j]) * g[j]
            g[i] = v / np.sqrt(v @ gram @ v)
        self.g, self.n, self.dim = g.astype(np.float64), n, dim

    def values(self, x):
        """[..., n] at reference points x [..., dim] (torch)."""
        m = torch.stack([math.prod((x[..., a] ** p[a] for a in range(self.dim)), start=torch.ones_like(x[..., 0]))
                         for p in self.mono], dim=-1)
        return m @ torch.as_tensor(self.g.T.copy(), device=x.device)

    def gradients(self, x):
        """[..., dim, n]"""
        rows = []
        for r in range(self.dim):
            rows.append(torch.stack([
                (p[r] * math.prod((x[..., a] ** (p[a] - (a == r)) for a in range(self.dim)),
                                  start=torch.ones_like(x[..., 0]))) if p[r] else torch.zeros_like(x[..., 0])
                for p in self.mono], dim=-1))
        return torch.stack(rows, dim=-2) @ torch.as_tensor(self.g.T.copy(), device=x.device)


# ---------------------------------------------------------------------------
# the step in plain torch, 64 bits


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


class Plain:
    """Geometry, fields and the SSP-RK3 step of one mesh and law, whole arrays."""

    def __init__(self, case, mesh, params):
        self.law, self.flux, self.dim, self.p, self.order = case["law"], case["flux"], case["dim"], params, case["order"]
        dev = self.dev = _device()
        v, cells, _ = mesh
        d = self.dim
        self.basis = _Basis(d, self.order)
        X = torch.as_tensor(v, device=dev)[:, :d]
        cv = torch.as_tensor(cells, device=dev)
        self.x0 = X[cv[:, 0]]
        nodes = [1, 2] if d == 2 else [3, 2, 1]
        self.J = torch.stack([X[cv[:, k]] - self.x0 for k in nodes], dim=1)  # [E, r, i] = d x_i / d xi_r
        self.Ji = torch.linalg.inv(self.J)                                   # [E, i, r]
        self.det = torch.linalg.det(self.J).abs()
        pair = [(a, b) for a in range(d + 1) for b in range(a)]
        ln = torch.stack([(X[cv[:, a]] - X[cv[:, b]]).norm(dim=1) for a, b in pair], dim=1)
        if d == 2:
            hp = 0.5 * ln.sum(dim=1)
            self.size = (hp * (hp - ln[:, 0]) * (hp - ln[:, 1]) * (hp - ln[:, 2])).sqrt() / hp * 2.0
        else:
            self.size = ln.min(dim=1).values
        xi, w = _tri_rule(max(1, 2 * self.order)) if d == 2 else _tet_rule(2 * self.order)
        self.xi = torch.as_tensor(xi, device=dev)
        self.w = torch.as_tensor(w, device=dev) * (0.5 if d == 2 else 1 / 6)
        self.phi, self.dphi = self.basis.values(self.xi), self.basis.gradients(self.xi)
        self.phi0 = float(self.basis.g[0, 0])
        corner = torch.as_tensor(np.vstack([np.zeros(d), np.eye(d)]), device=dev)
        self.phiv = self.basis.values(corner)
        # faces: left and right cell, points, the two sides' basis values
        f, key, o = _cell_faces(cells, d)
        k = key[o]
        first = np.ones(len(k), dtype=bool)
        first[1:] = k[1:] != k[:-1]
        at = np.flatnonzero(first)
        two = np.zeros(len(at), dtype=bool)
        two[:-1] = np.diff(at) == 2
        two[-1] = len(k) - at[-1] == 2
        E = len(cells)
        left, right = o[at] % E, np.where(two, o[np.minimum(at + 1, len(o) - 1)] % E, -1)
        perm = np.argsort(~two, kind="stable")  # interior faces first
        left, right, fv = left[perm], right[perm], f[o[at]][perm]
        self.ni = int(two.sum())
        self.eL = torch.as_tensor(left, device=dev)
        self.eR = torch.as_tensor(right[:self.ni], device=dev)
        P = X[torch.as_tensor(fv, device=dev)]                               # [F, dim, i]
        if d == 2:
            s, fw = np.polynomial.legendre.leggauss(self.order + 1)
            s, fw = torch.as_tensor((s + 1) / 2, device=dev), torch.as_tensor(fw / 2, device=dev)
            pts = P[:, None, 0] * (1 - s)[None, :, None] + P[:, None, 1] * s[None, :, None]
            e = P[:, 1] - P[:, 0]
            meas = e.norm(dim=1)
            n = torch.stack([e[:, 1], -e[:, 0]], dim=1) / meas[:, None]
        else:
            st, fw = _tri_rule(2 * self.order + 1)
            st, fw = torch.as_tensor(st, device=dev), torch.as_tensor(fw, device=dev)
            pts = (P[:, None, 0] * (1 - st.sum(dim=1))[None, :, None] + P[:, None, 1] * st[None, :, :1] +
                   P[:, None, 2] * st[None, :, 1:])
            c = torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
            meas = 0.5 * c.norm(dim=1)
            n = c / c.norm(dim=1, keepdim=True)
        mid = X[cv[self.eL]].mean(dim=1)
        out = ((pts.mean(dim=1) - mid) * n).sum(dim=1)
        self.n = torch.where(out[:, None] < 0, -n, n)
        self.jw = meas[:, None] * fw[None, :]
        at_ref = lambda e, x: torch.einsum("fqi,fir->fqr", x - self.x0[e][:, None], self.Ji[e])  # noqa: E731
        self.phiL = self.basis.values(at_ref(self.eL, pts))
        self.phiR = self.basis.values(at_ref(self.eR, pts[:self.ni]))
        self.bx = pts[self.ni:]

    # ---- fields and point physics
    def field(self, x, t):
        p = self.p
        if self.law == "scalar":  # the 2D pulse, constant along z on tets
            r2 = sum((x[..., i] - p[i] * t - p[3 + i]) ** 2 for i in range(2))
            return torch.exp(-r2 / p[6])[..., None]
        if self.law == "burgers":
            return (0.5 + p[9] * torch.sin(2 * math.pi * (x[..., 0] + x[..., 1])))[..., None]
        if self.law == "euler2d":
            b, dx, dy = p[8], x[..., 0] - (p[3] + t), x[..., 1] - (p[4] + t)
            e = torch.exp(0.5 * (1 - dx * dx - dy * dy))
            u, v = 1 - b / (2 * math.pi) * e * dy, 1 + b / (2 * math.pi) * e * dx
            rho = (1 - (GAMMA - 1) * b * b / (8 * GAMMA * math.pi ** 2) * e * e) ** (1 / (GAMMA - 1))
            return torch.stack([rho, rho * u, rho * v, rho ** GAMMA / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)], -1)
        if self.law == "euler3d":
            r2 = sum((x[..., i] - p[i] * t - p[3 + i]) ** 2 for i in range(3))
            rho = 1 + 0.2 * torch.exp(-r2 / p[6])
            k = 0.5 * (p[0] ** 2 + p[1] ** 2 + p[2] ** 2)
            return torch.stack([rho, rho * p[0], rho * p[1], 1 / (GAMMA - 1) + k * rho, rho * p[2]], -1)
        L = p[10]
        k, w = math.pi / L, math.pi * math.sqrt(2) / L
        sx, cx, sy, cy = (f(k * x[..., i]) for i in (0, 1) for f in (torch.sin, torch.cos))
        ez, hx, hy = sx * sy * math.cos(w * t), -(k / w) * sx * cy * math.sin(w * t), (k / w) * cx * sy * math.sin(w * t)
        z = torch.zeros_like(ez)
        return torch.stack([z, z, ez, hx, hy, z] if self.law == "maxwell3d" else [hx, hy, ez], -1)

    def _mom(self, U):
        return U[..., [1, 2]] if self.dim == 2 else U[..., [1, 2, 4]]

    def _pressure(self, U):
        return (GAMMA - 1) * (U[..., 3] - 0.5 * (self._mom(U) ** 2).sum(-1) / U[..., 0])

    def fluxes(self, U):
        """[..., field, direction]"""
        if self.law == "scalar":
            return U[..., None] * torch.as_tensor(self.p[:self.dim], device=U.device)
        if self.law == "burgers":
            return (0.5 * U * U)[..., None].expand(*U.shape, 2)
        if self.law in ("euler2d", "euler3d"):
            m, pr = self._mom(U), self._pressure(U)
            vel = m / U[..., :1]
            eye = torch.eye(self.dim, dtype=U.dtype, device=U.device)
            fm = m[..., :, None] * vel[..., None, :] + pr[..., None, None] * eye
            fe = (vel * (U[..., 3] + pr)[..., None])[..., None, :]
            rows = [m[..., None, :], fm[..., :2, :], fe] + ([fm[..., 2:, :]] if self.dim == 3 else [])
            return torch.cat(rows, dim=-2)
        z = torch.zeros_like(U[..., 0])
        if self.law == "maxwell2d":
            hx, hy, ez = U.unbind(-1)
            rows = [(z, ez), (-ez, z), (-hy, hx)]
        else:
            E, H = U[..., :3].unbind(-1), U[..., 3:].unbind(-1)
            rows = [(z, -H[2], H[1]), (H[2], z, -H[0]), (-H[1], H[0], z),
                    (z, E[2], -E[1]), (-E[2], z, E[0]), (E[1], -E[0], z)]
        return torch.stack([torch.stack(r, -1) for r in rows], -2)

    def normal_flux(self, U, n):
        return (self.fluxes(U) * n[..., None, :]).sum(-1)

    def numerical(self, n, L, R):
        if self.law == "scalar":
            vn = (n * torch.as_tensor(self.p[:self.dim], device=n.device)).sum(-1, keepdim=True)
            return vn * torch.where(vn > 0, L, R)
        if self.law == "burgers":
            return 0.5 * (self.normal_flux(L, n) + self.normal_flux(R, n))
        if self.law == "maxwell2d":
            # the interface state of the characteristic split, then its flux
            nx, ny = n[..., 0], n[..., 1]
            s, dl = 0.5 * (L + R), 0.5 * (L - R)
            hx = s[..., 0] * (nx * ny + ny * ny) + s[..., 1] * (nx * nx - nx * ny) + dl[..., 2] * ny
            hy = s[..., 0] * (ny * ny - nx * ny) + s[..., 1] * (nx * nx + nx * ny) - dl[..., 2] * nx
            return self.normal_flux(torch.stack([hx, hy, ny * dl[..., 0] - nx * dl[..., 1] + s[..., 2]], -1), n)
        if self.law == "maxwell3d":
            n3 = n.expand(*L.shape[:-1], 3)
            cr = lambda a: torch.linalg.cross(n3, a)  # noqa: E731
            E, H, dE, dH = 0.5 * (L + R)[..., :3], 0.5 * (L + R)[..., 3:], (R - L)[..., :3], (R - L)[..., 3:]
            return torch.cat([-cr(H) + 0.5 * cr(cr(dE)), cr(E) + 0.5 * cr(cr(dH))], -1)
        if self.flux == "godunov":
            return self._godunov(n, L, R)
        FL, FR = self.normal_flux(L, n), self.normal_flux(R, n)
        pL, pR = self._pressure(L), self._pressure(R)
        vL, vR = L[..., 1:3] / L[..., :1], R[..., 1:3] / R[..., :1]
        if self.flux == "llf":
            lam = torch.maximum((GAMMA * pL / L[..., 0]).sqrt() + (vL * n).sum(-1).abs(),
                                (GAMMA * pR / R[..., 0]).sqrt() + (vR * n).sum(-1).abs())
            return 0.5 * (FL + FR) - 0.5 * lam[..., None] * (R - L)
        # Roe
        a, b = L[..., 0].sqrt(), R[..., 0].sqrt()
        avg = lambda x, y: (x * a + y * b) / (a + b)  # noqa: E731
        u, v = avg(vL[..., 0], vR[..., 0]), avg(vL[..., 1], vR[..., 1])
        H = avg((L[..., 3] + pL) / L[..., 0], (R[..., 3] + pR) / R[..., 0])
        c = ((GAMMA - 1) * (H - 0.5 * (u * u + v * v))).sqrt()
        rho, nx, ny = a * b, n[..., 0], n[..., 1]
        vn = u * nx + v * ny
        dr, dp, du, dv = R[..., 0] - L[..., 0], pR - pL, vR[..., 0] - vL[..., 0], vR[..., 1] - vL[..., 1]
        dn = du * nx + dv * ny
        one, zero = torch.ones_like(vn), torch.zeros_like(vn)
        waves = [(vn.abs() * (dr - dp / (c * c)), (one, u, v, 0.5 * (u * u + v * v))),
                 (vn.abs() * (ny * du - nx * dv) * rho, (zero, ny * one, -nx * one, u * ny - v * nx)),
                 ((vn + c).abs() * 0.5 * (rho * dn / c + dp / (c * c)), (one, u + c * nx, v + c * ny, H + c * vn)),
                 ((vn - c).abs() * 0.5 * (-rho * dn / c + dp / (c * c)), (one, u - c * nx, v - c * ny, H - c * vn))]
        diss = sum(s[..., None] * torch.stack([x.expand(s.shape) for x in r], -1) for s, r in waves)
        return 0.5 * (FL + FR - diss)

    def _godunov(self, n, L, R):
        """Flux of the exact Riemann solution on the face (Newton on the star pressure)."""
        n = n.expand(*L.shape[:-1], self.dim)

        def prim(U):
            v = self._mom(U) / U[..., :1]
            un = (v * n).sum(-1)
            return U[..., 0], un, v - un[..., None] * n, self._pressure(U)

        (rl, ul, tl, pl), (rr, ur, tr, pr) = prim(L), prim(R)
        g, cl, cr = GAMMA, (GAMMA * pl / rl).sqrt(), (GAMMA * pr / rr).sqrt()

        def side(p, r, pk, c):
            A, B = 2 / ((g + 1) * r), (g - 1) / (g + 1) * pk
            q = (A / (p + B)).sqrt()
            x = (p / pk) ** ((g - 1) / (2 * g))
            f = torch.where(p > pk, (p - pk) * q, 2 * c / (g - 1) * (x - 1))
            df = torch.where(p > pk, q * (1 - 0.5 * (p - pk) / (p + B)), x * c / (g * p))
            return f, df

        p = (0.5 * (pl + pr) - 0.125 * (ur - ul) * (rl + rr) * (cl + cr)).clamp_min(1e-14)
        for _ in range(14):
            (fl, dl), (fr, dr) = side(p, rl, pl, cl), side(p, rr, pr, cr)
            p = (p - (fl + fr + ur - ul) / (dl + dr)).clamp_min(1e-14)
        us = 0.5 * (ul + ur + side(p, rr, pr, cr)[0] - side(p, rl, pl, cl)[0])
        lft = us >= 0
        sg = torch.where(lft, 1.0, -1.0)
        r0, u0, p0, c0 = (torch.where(lft, a, b) for a, b in ((rl, rr), (ul, ur), (pl, pr), (cl, cr)))
        C = (g - 1) / (g + 1)
        y = p / p0
        shock = p >= p0
        rs = r0 * torch.where(shock, (y + C) / (C * y + 1), y ** (1 / g))
        # sampled as DG-Parallel does: a flow supersonic on both sides keeps its
        # upwind state, a shock gives the star state, a rarefaction the star
        # state or the sonic point of its fan
        ahead = torch.where(lft, (ul >= cl) & (ur >= cr), (ul <= -cl) & (ur <= -cr))
        behind = shock | ((us - sg * (g * p / rs).sqrt()) * us <= 0)
        k = (2 / (g + 1) + sg * (g - 1) / (g + 1) * u0 / c0).clamp_min(1e-30)
        pick = lambda a, b, c: torch.where(ahead, a, torch.where(behind, b, c))  # noqa: E731
        rho, un, pr_ = pick(r0, rs, r0 * k ** (2 / (g - 1))), pick(u0, us, sg * c0 * k), \
            pick(p0, p, p0 * k ** (2 * g / (g - 1)))
        vel = un[..., None] * n + torch.where(lft[..., None], tl, tr)
        en = pr_ / (g - 1) + 0.5 * rho * (vel * vel).sum(-1)
        m = rho[..., None] * vel
        U = torch.cat([rho[..., None], m[..., :2], en[..., None]] + ([m[..., 2:]] if self.dim == 3 else []), -1)
        return self.normal_flux(U, n)

    # ---- the operator
    def project(self, t=0.0):
        x = self.x0[:, None] + torch.einsum("qr,eri->eqi", self.xi, self.J)
        return torch.einsum("eqj,qk,q->ejk", self.field(x, t), self.phi, self.w).contiguous()

    def rhs(self, c, t):
        U = torch.einsum("qk,ejk->eqj", self.phi, c)
        G = torch.einsum("eqji,eir->eqjr", self.fluxes(U), self.Ji) * (self.det[:, None] * self.w)[..., None, None]
        r = torch.einsum("eqjr,qrk->ejk", G, self.dphi)
        ni, n = self.ni, self.n[:, None, :]
        UL = torch.einsum("fqk,fjk->fqj", self.phiL, c[self.eL])
        UR = torch.einsum("fqk,fjk->fqj", self.phiR, c[self.eR])
        Fi = self.numerical(n[:ni], UL[:ni], UR)
        Ub, nb = UL[ni:], n[ni:]
        if self.law == "maxwell3d":  # perfect conductor
            ghost = torch.cat([-Ub[..., :3], Ub[..., 3:]], -1)
        else:
            ghost = self.field(self.bx, t)
        if self.law == "burgers":  # inflow and outflow by the sign of the interior flux
            own, far = self.normal_flux(Ub, nb), self.normal_flux(ghost, nb)
            Fb = torch.where(own < 0, far, own)
        else:
            Fb = self.numerical(nb, Ub, ghost)
        F = torch.cat([Fi, Fb]) * self.jw[..., None]
        r = r.index_add(0, self.eL, -torch.einsum("fqj,fqk->fjk", F, self.phiL))
        return r.index_add(0, self.eR, torch.einsum("fqj,fqk->fjk", F[:ni], self.phiR))

    def speed(self, U):
        if self.law == "scalar":
            return torch.full_like(U[..., 0], sum(abs(a) for a in self.p[:3]))
        if self.law in ("euler2d", "euler3d"):
            return (GAMMA * self._pressure(U) / U[..., 0]).sqrt() + (self._mom(U) / U[..., :1]).norm(dim=-1)
        return torch.ones_like(U[..., 0])

    def dt(self, c):
        a = self.speed(c[:, :, 0] * self.phi0)
        if self.dim == 2:
            a = torch.maximum(a, self.speed(torch.einsum("qk,ejk->eqj", self.phiv, c)).max(dim=1).values)
        return float((self.size * CFL / (a * (2 * self.order + 1))).min())

    def step(self, u, t, dt):
        k = dt / self.det[:, None, None]
        u1 = u + k * self.rhs(u, t)
        u2 = 0.25 * (u1 + k * self.rhs(u1, t + dt) + 3 * u)
        return (2 * (u2 + k * self.rhs(u2, t + 0.5 * dt)) + u) / 3

    def run(self, u, steps):
        t = 0.0
        for _ in range(steps):
            dt = self.dt(u)
            u = self.step(u, t, dt)
            t += dt
        return u


# ---------------------------------------------------------------------------
# the cases


def _params(case, rng):
    law = case["law"]
    jit = lambda s: float(rng.uniform(-s, s))  # noqa: E731
    if law == "scalar":
        return dgp.law_params(velocity=(1.0, 0.5, 0.0 if case["dim"] == 2 else 0.25),
                              center=(0.3 + jit(0.05), 0.3 + jit(0.05), 0.0), width=0.05)
    if law == "burgers":
        return dgp.law_params(amplitude=0.25 + jit(0.1))
    if law == "euler2d":
        return dgp.law_params(velocity=(1.0, 1.0, 0.0), center=(5.0 + jit(0.5), 5.0 + jit(0.5), 0.0), gamma=GAMMA,
                              beta=5.0 + jit(0.2))
    if law == "euler3d":
        return dgp.law_params(velocity=(1.0, 0.5, 0.25), center=(0.5 + jit(0.1), 0.5 + jit(0.1), 0.5), width=0.05,
                              gamma=GAMMA)
    return dgp.law_params(cavity=1.0)


def _mesh(case, rng):
    if case["dim"] == 3:
        return _tet_mesh(case["nx"], _box(case["law"]), rng)
    return _tri_mesh(case["nx"], case["ny"], _box(case["law"]), rng, case.get("ratio"))


def _inputs(case, seed):
    """(mesh, law parameters, initial state) of one problem from its seed."""
    rng = np.random.default_rng(seed)
    mesh = _mesh(case, rng)
    params = _params(case, rng)
    plain = Plain(case, mesh, params)
    state = plain.project(0.0)
    if case["law"].startswith("maxwell"):  # the cavity mode with a second one of random strength per field
        a = torch.as_tensor(rng.uniform(0.1, 0.3, state.shape[1]), device=state.device)
        state = state + a[None, :, None] * state[:, 2:3, :]
    return rng, mesh, params, plain, state


def _dgp_mesh(case, mesh):
    v, cells, bf = mesh
    tag = 40000 if case["law"] == "maxwell3d" else 1
    return dgp.Mesh.from_arrays(case["dim"], v, cells, 100, bf, np.full(len(bf), tag))


def _law(case, params):
    field = FIELDS[case["law"]]
    return dgp.Law(LAWS[case["law"]], FLUXES[case["flux"]], field, params)


def _solver(case, mesh, params):
    return dgp.Solver(_dgp_mesh(case, mesh), _law(case, params), case["order"],
                      dgp.MIXED if case["mixed"] else dgp.FP64,
                      rule=dgp.RULE_WORKLOAD if case["workload_rule"] else dgp.RULE_REFERENCE)


def _batch(case, seed):
    """Sizes, orders and amplitudes of a batch, log-uniform between nx and ny cells."""
    rng = np.random.default_rng(seed)
    out = []
    # the batch's sizes are the case's; meshes and amplitudes are the seed's
    shape = np.random.default_rng(case["count"] * 7919 + case["nx"])
    for i in range(case["count"]):
        n = int(round(math.sqrt(math.exp(shape.uniform(math.log(case["nx"]), math.log(case["ny"]))) / 2)))
        out.append({"nx": n, "order": 1 + i % case["order"], "amplitude": float(rng.uniform(0.5, 1.5)),
                    "mesh": _tri_mesh(n, n, 1.0, rng)})
    return out


ADJOINT_DT = {"euler2d": 0.02, "scalar": 0.03}


def _adjoint_dt(case):
    return ADJOINT_DT[case["law"]] * _box(case["law"]) / (max(case["nx"], case["ny"]) * (2 * case["order"] + 1) * 3)


def _receivers(case, rng):
    b = _box(case["law"])
    x = rng.uniform(0.2 * b, 0.8 * b, (case["receivers"], 2))
    return x, rng.uniform(0.7, 1.0, case["receivers"])


def prepare(case, seed):
    if case["do"] == "ensemble":
        batch = _batch(case, seed)
        meshes = [_dgp_mesh(case, b["mesh"]) for b in batch]
        laws = [_law(case, dgp.law_params(amplitude=b["amplitude"])) for b in batch]
        e = dgp.Ensemble(meshes, laws, [b["order"] for b in batch], dgp.FP64, dgp.LIMITER_MOMENT)
        return {"case": case, "ensemble": e}
    rng, mesh, params, _, state = _inputs(case, seed)
    s = _solver(case, mesh, params)
    st = {"case": case, "solver": s}
    if case["do"] == "step":
        st["host"] = state.cpu().numpy()
        st["host_out"] = np.empty_like(st["host"])
        st["dt"] = 0.1 * _box(case["law"]) / (max(case["nx"], case["ny"]) * (2 * case["order"] + 1) * 6)
        return st
    if case["do"] == "adjoint":
        s.set_receivers(*_receivers(case, rng))
        st["dt"] = _adjoint_dt(case)
    elif case["do"] == "lts":
        s.set_p0_fallback(False)
        s.set_time_stepping(dgp.STEPPING_LOCAL)
    st["state"] = state
    st["out"] = torch.empty_like(state)
    torch.cuda.synchronize()  # the solver reads the state on its own stream
    return st


def run(state):
    case = state["case"]
    if case["do"] == "ensemble":
        e = state["ensemble"]
        e.project(0.0)
        t, steps, _, _ = e.run(0.0, 0.0, CFL, max_steps=case["steps"])
        return {"t": t, "steps": steps, "states": [e.get_state(i) for i in range(e.n)]}
    s = state["solver"]
    if case["do"] == "step":
        s.set_state(state["host"])
        resid = s.step(0.0, state["dt"])
        return {"state": s.get_state(state["host_out"]), "resid": resid}
    s.set_state_device(state["state"].data_ptr())
    if case["do"] == "adjoint":
        j = s.forward_checkpointed(0.0, state["dt"], case["steps"], case["every"])
        return {"objective": j, "gradient": s.backward()}
    t, steps = s.run(0.0, 0.0, CFL, max_steps=case["steps"])
    s.get_state_device(state["out"].data_ptr())
    # the mixed form's right-hand side carries 32 bits: its solution is kept in them
    u = state["out"].float() if case["mixed"] else state["out"]
    return {"t": t, "steps": steps, "state": u}


def _shape(case):
    """(cells, faces, fields, modes, volume points, face points) of a single problem."""
    p, d = case["order"], case["dim"]
    if d == 2:
        E = 2 * case["nx"] * case["ny"]
        F = E + E // 2 + case["nx"] + case["ny"]
        return E, F, NFIELDS[case["law"]], (p + 1) * (p + 2) // 2, (1, 3, 6, 12, 16)[p], p + 1
    E = 6 * case["nx"] ** 3
    return (E, 2 * E + 6 * case["nx"] ** 2, NFIELDS[case["law"]], (p + 1) * (p + 2) * (p + 3) // 6,
            (1, 4, 11 if case["workload_rule"] else 14)[p], (1, 4, 6 if case["workload_rule"] else 7)[p])


def _stage_work(E, F, M, N, nq, nqf, d):
    """One stage: the state in and out (u_n in two of three) and the geometry;
    interpolation, flux, contraction, traces, Riemann fluxes and lift."""
    b = E * ((2 + 2 / 3) * M * N * 8 + (d * d + 1) * 8) + F * (8 * d + 8 + 10)
    f = E * (2 * M * N * nq * (1 + d) + nq * M * (10 + 2 * d * d)) + F * nqf * (8 * M * N + 30 * M)
    return np.array([b, f])


def work(case):
    d = case["dim"]
    if case["do"] == "ensemble":
        total = np.zeros(2)
        for b in _batch(case, 0):
            one = dict(case, nx=b["nx"], ny=b["nx"], order=b["order"])
            sh = _shape(one)
            # the stages and the limiter's pass over the state after each
            total += 3 * case["steps"] * (_stage_work(*sh, d) + np.array([16.0 * sh[0] * sh[3], 30.0 * sh[0] * sh[3]]))
        return {"bytes": float(total[0]), "flops": float(total[1])}
    sh = _shape(case)
    stage = _stage_work(*sh, d)
    io = np.array([4.0 * 8 * sh[0] * sh[2] * sh[3], 0.0])
    stages = 3 * case["steps"]
    if case["do"] == "adjoint":  # forward, (recompute,) and reversed stages at about twice a forward one
        stages *= (1 if case["every"] == 0 else 2) + 2
    elif case["do"] == "lts":  # two stages per substep; a quarter of the cells, about, in each of four bins
        stages = case["steps"] * 2 * 3.75
    total = stages * stage + io
    return {"bytes": float(total[0]), "flops": float(total[1])}


def exact(case, seed):
    # the limiter's switches and the local steps' bookkeeping have no closed
    # 64-bit counterpart here: those passes are compared as they are
    if case["do"] in ("ensemble", "lts"):
        return None
    with torch.no_grad():
        rng, mesh, params, plain, u0 = _inputs(case, seed)
        if case["do"] == "step":
            dt = 0.1 * _box(case["law"]) / (max(case["nx"], case["ny"]) * (2 * case["order"] + 1) * 6)
            u = plain.step(u0, 0.0, dt)
            return {"state": u.cpu().numpy(), "resid": float(((u - u0) ** 2).sum())}
        if case["do"] == "run":
            return {"t": None, "steps": None, "state": plain.run(u0, case["steps"])}
    x, obs = _receivers(case, rng)
    x, obs = torch.as_tensor(x, device=u0.device), torch.as_tensor(obs, device=u0.device)
    cell, phi = [], []
    for i in range(len(x)):
        xi = torch.einsum("ei,eir->er", x[i] - plain.x0, plain.Ji)
        inside = torch.minimum(xi.min(dim=1).values, 1 - xi.sum(dim=1))
        cell.append(inside.argmax())
        phi.append(plain.basis.values(xi[cell[-1]]))
    cell, phi = torch.stack(cell), torch.stack(phi)
    dt = _adjoint_dt(case)
    states = [u0]
    with torch.no_grad():
        for k in range(case["steps"]):
            states.append(plain.step(states[-1], k * dt, dt))
    u = states[-1].clone().requires_grad_()
    j = (((phi * u[cell, 0]).sum(dim=1) - obs) ** 2).sum()
    (lam,) = torch.autograd.grad(j, u)
    for k in reversed(range(case["steps"])):  # one step's graph at a time
        u = states[k].clone().requires_grad_()
        (lam,) = torch.autograd.grad(plain.step(u, k * dt, dt), u, grad_outputs=lam)
    return {"objective": float(j.detach()), "gradient": lam.cpu().numpy()}
