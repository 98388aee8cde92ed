"""The adjoint's row, point and flux mapping at the sizes where it can go wrong
(one cell more or less than a tile, odd mode counts, laws of one to six fields)
and the Roe flux's reverse pass on states with jumps: the gradient of a seeded
linear functional of the state after two steps, against central differences of
the same forward map along a random direction.

The differences' own error bounds the tolerance.  Linear laws have no
truncation: eps = 1e-2, rounding 1e-16 / eps of the functional, 1e-9 covers it by
four orders.  The others: eps = 1e-6, truncation eps^2, rounding 1e-10 (the
functional's terms cancel by about ten), and an eps small enough that hardly a
point's switch (the larger speed, a wave's sign) lies inside it: 1e-6."""
import numpy as np
import pytest

import dgp
from dgp import meshgen
from cases import SCALAR2D, SINE, TM110, VORTEX
from test_stage_rows import _mesh

LAWS = {
    "scalar": (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, SCALAR2D, 1.0, 1e-9),
    "burgers": (dgp.LAW_BURGERS2D, dgp.FLUX_LLF, dgp.FIELD_SINE, SINE, 1.0, 1e-6),
    "maxwell2d": (dgp.LAW_MAXWELL2D, dgp.FLUX_UPWIND, dgp.FIELD_TM2D, TM110, 1.0, 1e-9),
    "maxwell3d": (dgp.LAW_MAXWELL3D, dgp.FLUX_UPWIND, dgp.FIELD_TM110, TM110, 1.0, 1e-9),
    "roe": (dgp.LAW_EULER2D, dgp.FLUX_ROE, dgp.FIELD_VORTEX, VORTEX, 10.0, 1e-6),
    "llf": (dgp.LAW_EULER2D, dgp.FLUX_LLF, dgp.FIELD_VORTEX, VORTEX, 10.0, 1e-6),
}


@pytest.mark.gpu
@pytest.mark.parametrize("every", [0, 1])
@pytest.mark.parametrize("kind,order,cells", [("scalar", 1, 129), ("scalar", 4, 127), ("burgers", 2, 129),
                                              ("maxwell2d", 2, 43), ("maxwell3d", 2, 0), ("roe", 0, 65),
                                              ("roe", 1, 33), ("roe", 2, 31), ("roe", 4, 65), ("llf", 3, 33)])
def test_adjoint_rows_match_central_differences(kind, order, cells, every):
    law, flux, field, prm, box, tol = LAWS[kind]
    m = _mesh(kind, cells, box)
    mesh = dgp.Mesh.from_arrays(m.dim, m.vertices, m.cells, 100, m.bfaces, m.btags)
    s = dgp.Solver(mesh, dgp.Law(law, flux, field, prm), order)
    s.set_receivers(m.vertices[m.cells[0]].mean(axis=0)[None, :m.dim], np.array([0.5]))
    rng = np.random.default_rng(4)
    u0 = s.get_state()
    if kind in ("roe", "llf"):  # jumps of a few percent between neighbours
        u0 = u0 * (1.0 + 0.03 * rng.normal(size=(len(u0), u0.shape[1], 1)))
    s.set_state(u0)
    dt = 0.2 * s.cfl_dt(0.1)
    seed = rng.normal(size=u0.shape)
    d = rng.normal(size=u0.shape) * np.abs(u0[:, :, :1]).mean()

    def value(u):
        s.set_state(u)
        s.forward_checkpointed(0.1, dt, 2, every)
        return float((seed * s.get_state()).sum())

    value(u0)
    g = float((s.backward(seed) * d).sum())
    eps = 1e-2 if tol < 1e-8 else 1e-6
    fd = (value(u0 + eps * d) - value(u0 - eps * d)) / (2 * eps)
    scale = float(np.linalg.norm(seed) * np.linalg.norm(d))
    assert abs(g - fd) <= tol * max(abs(g), 1e-3 * scale)
