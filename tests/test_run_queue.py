"""Runs whose step graphs are queued ahead of the host: the step count, time and
state are those of single steps whichever of the step limit and the end time
comes first, for counts below, at and beyond what is queued at once (eight graphs
of eight steps, four in an ensemble), and a time step that is not positive ends
the run with an error at the graph it appears in.

A run and single steps take the same arithmetic but for the order of the CFL
reduction's inputs (none in a minimum): states to 1e-13 of the largest value,
times to 1e-14.  Ensembles equal their single solvers bit for bit."""
import math

import numpy as np
import pytest

import dgp
from dgp import meshgen
from cases import SCALAR2D, params, rel

pytestmark = pytest.mark.gpu


def _mesh(n, seed=5):
    m = meshgen.tri_square(n, n, seed=seed)
    return dgp.Mesh.from_arrays(m.dim, m.vertices, m.cells, 100, m.bfaces, m.btags)


def _steps(s, u0, cfl, tend, max_steps):
    s.set_state(u0)
    t, n = 0.0, 0
    while not (max_steps and n >= max_steps) and not (tend > 0 and t >= tend):
        dt = s.cfl_dt(cfl)
        if tend > 0:
            dt = (tend - t) / math.ceil((tend - t) / dt)
        s.step(t, dt)
        t, n = t + dt, n + 1
    return t, n, s.get_state()


@pytest.mark.parametrize("max_steps,tend_steps", [(3, 0), (8, 0), (13, 0), (64, 0), (75, 0), (5, 40.5), (13, 40.5),
                                                  (43, 20.5), (75, 11.5), (0, 5.5), (0, 43.5)])
def test_run_equals_single_steps(max_steps, tend_steps):
    s = dgp.Solver(_mesh(9), dgp.Law(dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, SCALAR2D), 1)
    u0 = s.get_state()
    tend = tend_steps * s.cfl_dt(0.1)
    t1, n1, u1 = _steps(s, u0, 0.1, tend, max_steps)
    s.set_state(u0)
    t, n = s.run(0.0, tend, 0.1, max_steps)
    assert n == n1 and abs(t - t1) <= 1e-14 * t1
    assert rel(s.get_state(), u1) < 1e-13


@pytest.mark.parametrize("max_steps,tend", [(8, 0.0), (13, 0.0), (43, 0.0), (13, 10.0), (43, 0.02), (3, 10.0)])
def test_ensemble_equals_single_solvers_under_a_step_limit(max_steps, tend):
    meshes = [_mesh(n, seed=n) for n in (5, 9, 7)]
    laws = [dgp.Law(dgp.LAW_BURGERS2D, dgp.FLUX_LLF, dgp.FIELD_SINE, params(amplitude=a)) for a in (0.5, 0.9, 1.2)]
    orders = [1, 3, 1]
    e = dgp.Ensemble(meshes, laws, orders)
    e.project(0.0)
    t, n, _, _ = e.run(0.0, tend, 0.1, max_steps)
    for i in range(3):
        s = dgp.Solver(meshes[i], laws[i], orders[i])
        s.project(0.0)
        ts, ns = s.run(0.0, tend, 0.1, max_steps)
        assert n[i] == ns and abs(t[i] - ts) <= 1e-14 * ts
        assert np.array_equal(e.get_state(i), s.get_state())


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("max_steps,stops", [(3, 1), (9, 8), (16, 8), (64, 8), (70, 8)])
def test_step_that_is_not_positive_ends_a_run(max_steps, stops, fused):
    """A speed that overflows gives a step of zero.  The run ends where the host
    would have found it between two graphs, and the graphs behind leave the
    state alone; a run of exactly one graph ends by its step limit first."""
    prm = params(velocity=(1e308, 1e308, 0.0), center=(0.3, 0.3, 0.0), width=0.01)
    s = dgp.Solver(_mesh(6), dgp.Law(dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, prm), 1)
    s.set_fused(fused)
    u0 = s.get_state()
    assert s.run(0.0, 0.0, 0.1, stops) == (0.0, stops)
    u1 = s.get_state()
    s.set_state(u0)
    with pytest.raises(dgp.DGPError) as ei:
        s.run(0.0, 0.0, 0.1, max_steps)
    assert ei.value.code == -5
    assert np.array_equal(s.get_state(), u1, equal_nan=True)
    # the next run starts afresh
    s.set_state(u0)
    assert s.run(0.0, 0.0, 0.1, stops)[1] == stops
