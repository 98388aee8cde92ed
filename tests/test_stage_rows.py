"""The fused stage kernel's row and point mapping at the sizes where it can go
wrong: cell counts that leave the last tile with an odd number of rows or of
values (no bulk copy), one face point per face (P0), odd mode counts, a tile's
worth of cells and one more or less, laws of one to six fields, periodic
partners -- right-hand side, CFL step and three steps against the oracle.

Tolerances as everywhere between the CUDA FP64 form and the oracle: states
1e-12, right-hand sides 1e-11 relative to the largest value; states of the
mixed form 2e-5.  The mixed form's right-hand side is not compared by itself:
its error is FP32 rounding of its terms, which cancel in it without a bound
(the separate kernels' differ by 6e-5 of the 3D pulse's right-hand side)."""
import numpy as np
import pytest

import dgp
from dgp import meshgen
from cases import PULSE3D, SCALAR2D, SCALAR3D, SCALAR_PERIODIC, SINE, TM110, VORTEX, rel
from oracle_bind import Oracle

LAWS = {
    "scalar": (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, SCALAR2D, 1.0),
    "burgers": (dgp.LAW_BURGERS2D, dgp.FLUX_LLF, dgp.FIELD_SINE, SINE, 1.0),
    "maxwell2d": (dgp.LAW_MAXWELL2D, dgp.FLUX_UPWIND, dgp.FIELD_TM2D, TM110, 1.0),
    "euler": (dgp.LAW_EULER2D, dgp.FLUX_ROE, dgp.FIELD_VORTEX, VORTEX, 10.0),
    "scalar3d": (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS3D, SCALAR3D, 1.0),
    "euler3d": (dgp.LAW_EULER3D, dgp.FLUX_GODUNOV, dgp.FIELD_PULSE3D, PULSE3D, 1.0),
    "maxwell3d": (dgp.LAW_MAXWELL3D, dgp.FLUX_UPWIND, dgp.FIELD_TM110, TM110, 1.0),
}

# triangles: 2 nx ny cells cut to `cells`; 33 and 65 leave one cell (Euler
# tiles hold 32), 127 and 129 frame a one-field tile, 43 a three-field one
CASES = [("scalar", 0, 129), ("scalar", 1, 127), ("scalar", 4, 129), ("burgers", 1, 129), ("burgers", 4, 127),
         ("maxwell2d", 1, 43), ("maxwell2d", 4, 85), ("euler", 0, 33), ("euler", 1, 65), ("euler", 2, 31),
         ("euler", 4, 33), ("scalar3d", 1, 0), ("scalar3d", 3, 0), ("euler3d", 2, 0), ("maxwell3d", 0, 0),
         ("maxwell3d", 3, 0)]


def _mesh(kind, cells, box):
    if kind.endswith("3d"):
        return meshgen.tet_cube(3, seed=3, boundary_tag=40000 if kind == "maxwell3d" else 1)
    m = meshgen.tri_square(11, 6, 0.0, box, 0.0, box, seed=5)
    c = m.cells[:cells]
    # the boundary of what is left: edges that belong to one cell
    e = np.sort(np.concatenate([c[:, [0, 1]], c[:, [1, 2]], c[:, [2, 0]]]), axis=1)
    u, n = np.unique(e, axis=0, return_counts=True)
    used = np.unique(c)
    new = np.full(len(m.vertices), -1)
    new[used] = np.arange(len(used))
    b = u[n == 1]
    return meshgen.Mesh(2, m.vertices[used], new[c], new[b], np.ones(len(b), dtype=np.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [dgp.FP64, dgp.MIXED])
@pytest.mark.parametrize("kind,order,cells", CASES)
def test_rows_and_points_match_oracle(tmp_path, kind, order, cells, precision):
    law, flux, field, prm, box = LAWS[kind]
    msh = str(tmp_path / "m.msh")
    m = _mesh(kind, cells, box)
    assert m.num_cells == (cells or 162)
    meshgen.write_msh_v1(m, msh)
    o = Oracle(msh, law, flux, order, field, prm)
    s = dgp.Solver(dgp.Mesh.from_msh(msh), dgp.Law(law, flux, field, prm), order, precision)
    s.set_fused(True)
    ts = 1e-12 if precision == dgp.FP64 else 2e-5
    u0 = o.state()
    s.set_state(u0)
    if precision == dgp.FP64:
        assert rel(s.rhs(0.2), o.rhs(0.2)) < 1e-11
    t = 0.0
    for _ in range(3):
        dt = o.cfl_dt(0.1)
        rg, ro = s.step(t, dt), o.step(t, dt)
        t += dt
        if precision == dgp.FP64:
            assert abs(rg - ro) <= 1e-10 * ro
    assert rel(s.get_state(), o.state()) < ts
    # the step that the last stage reduced for the next one
    s.set_state(u0)
    tg, n = s.run(0.0, 0.0, 0.1, 3)
    assert n == 3 and abs(tg - t) <= (1e-13 if precision == dgp.FP64 else 2e-5) * t


@pytest.mark.gpu
@pytest.mark.parametrize("order", [1, 2, 4])
def test_periodic_partner_rows_match_oracle(tmp_path, order):
    msh = str(tmp_path / "p.msh")
    meshgen.write_msh_v1(meshgen.tri_square(9, 9, -1.0, 1.0, -1.0, 1.0, jitter=0.0, side_tags=(610, 510, 610, 510)),
                         msh)
    args = (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, SCALAR_PERIODIC)
    o = Oracle(msh, *args[:2], order, *args[2:])
    s = dgp.Solver(dgp.Mesh.from_msh(msh), dgp.Law(*args[:3], args[3]), order)
    s.set_fused(True)
    assert rel(s.rhs(0.0), o.rhs(0.0)) < 1e-11
    dt = o.cfl_dt(0.1)
    s.step(0.0, dt)
    o.step(0.0, dt)
    assert rel(s.get_state(), o.state()) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("kind,jump", [("godunov", 1e-3), ("godunov", 1.0), ("euler3d", 0.1), ("euler3d", 1.0)])
def test_exact_riemann_of_random_jumps_matches_oracle(tmp_path, kind, jump, fused):
    """Piecewise constant states with jumps of every size between neighbours:
    weak waves take riemann_face's short path, strong ones the full iteration.
    The flux is the oracle's to rounding, so the right-hand side is to 1e-11."""
    dim = 3 if kind == "euler3d" else 2
    law, flux, field, prm, box = LAWS["euler3d"] if dim == 3 else \
        (dgp.LAW_EULER2D, dgp.FLUX_GODUNOV, dgp.FIELD_VORTEX, VORTEX, 10.0)
    msh = str(tmp_path / "m.msh")
    meshgen.write_msh_v1(_mesh(kind, 129, box), msh)
    o = Oracle(msh, law, flux, 0, field, prm)
    s = dgp.Solver(dgp.Mesh.from_msh(msh), dgp.Law(law, flux, field, prm), 0)
    s.set_fused(fused)
    rng = np.random.default_rng(11)
    u = o.state()
    n = len(u)
    phi0 = np.sqrt(2.0 if dim == 2 else 6.0)
    rho, pr = np.exp(0.5 * jump * rng.normal(size=n)), np.exp(jump * rng.normal(size=n))
    v = 0.3 + 0.8 * jump * rng.normal(size=(n, dim))
    u[:, 0, 0] = rho
    u[:, 1, 0], u[:, 2, 0] = rho * v[:, 0], rho * v[:, 1]
    if dim == 3:
        u[:, 4, 0] = rho * v[:, 2]
    u[:, 3, 0] = pr / 0.4 + 0.5 * rho * (v ** 2).sum(axis=1)
    u /= phi0
    o.set_state(u)
    s.set_state(u)
    assert rel(s.rhs(0.1), o.rhs(0.1)) < 1e-11
