"""The exact Riemann solver in the mixed form's FP32 on piecewise constant states
with jumps between neighbours from a tenth to factors of thousands in pressure:
short path, full iteration, shocks and fans.

At P0 there is no volume term, and the right-hand side is a sum of face fluxes.
A flux carries some thirty roundings of 6e-8, amplified by up to ten in the
pressure's difference: 2e-5 of the fluxes, which the largest right-hand side
reaches for jumps of one and more and stays below in proportion for smaller
ones (fluxes of the common state cancel).  Where the solver's twelve iterations
end without a value in FP64 too (two faces of the largest jumps on tets), there
is nothing to compare."""
import numpy as np
import pytest

import dgp
from dgp import meshgen
from cases import rel
from oracle_bind import Oracle
from test_stage_rows import LAWS, VORTEX, _mesh


@pytest.mark.gpu
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("jump", [0.1, 1.0, 3.0])
@pytest.mark.parametrize("kind", ["godunov", "euler3d"])
def test_mixed_riemann_of_random_jumps_matches_oracle(tmp_path, kind, jump, fused):
    dim = 3 if kind == "euler3d" else 2
    law, flux, field, prm, box = LAWS["euler3d"] if dim == 3 else \
        (dgp.LAW_EULER2D, dgp.FLUX_GODUNOV, dgp.FIELD_VORTEX, VORTEX, 10.0)
    msh = str(tmp_path / "m.msh")
    meshgen.write_msh_v1(_mesh(kind, 129, box), msh)
    o = Oracle(msh, law, flux, 0, field, prm)
    s = dgp.Solver(dgp.Mesh.from_msh(msh), dgp.Law(law, flux, field, prm), 0, dgp.MIXED)
    s.set_fused(fused)
    rng = np.random.default_rng(12)
    u = o.state()
    n = len(u)
    rho, pr = np.exp(0.5 * jump * rng.normal(size=n)), np.exp(jump * rng.normal(size=n))
    v = 0.3 + 0.8 * min(jump, 1.0) * rng.normal(size=(n, dim))
    u[:, 0, 0] = rho
    u[:, 1, 0], u[:, 2, 0] = rho * v[:, 0], rho * v[:, 1]
    if dim == 3:
        u[:, 4, 0] = rho * v[:, 2]
    u[:, 3, 0] = pr / 0.4 + 0.5 * rho * (v ** 2).sum(axis=1)
    u /= np.sqrt(2.0 if dim == 2 else 6.0)
    o.set_state(u)
    s.set_state(u)
    want = o.rhs(0.1)
    has = np.isfinite(want).all(axis=(1, 2))
    assert has.sum() >= n - 4
    assert rel(s.rhs(0.1)[has], want[has]) < 2e-5 * max(1.0, 1.0 / jump)
