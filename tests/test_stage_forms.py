"""The two stage forms' tiles: the element kernel and the face slots have their
own tile size, ensembles start their instances on the tiles of the form they
run, and both forms give what single solvers give."""
import numpy as np
import pytest

import dgp
from dgp import meshgen
from test_zz_no_alloc import rhs_noalloc
from cases import PULSE3D, SCALAR2D, SCALAR3D, SINE, TM110, VORTEX, rel

pytestmark = pytest.mark.gpu


def _mesh(dim, n, seed, tag=1, box=1.0):
    m = meshgen.tet_cube(n, seed=seed, boundary_tag=tag) if dim == 3 else \
        meshgen.tri_square(n, n, 0.0, box, 0.0, box, seed=seed)
    return dgp.Mesh.from_arrays(m.dim, m.vertices, m.cells, 100, m.bfaces, m.btags)


# cells of a tile: the element kernel's, at most 64 KB, and the stage kernel's,
# at most 96 KB or a row a thread
@pytest.mark.parametrize("kind,order,elem,stage", [("maxwell3d", 2, 14, 21), ("maxwell3d", 3, 8, 12),
                                                   ("euler3d", 2, 17, 25), ("euler", 4, 25, 32), ("euler", 3, 32, 32)])
def test_forms_have_their_own_tiles(kind, order, elem, stage):
    args = {"maxwell3d": (dgp.LAW_MAXWELL3D, dgp.FLUX_UPWIND, dgp.FIELD_TM110, TM110),
            "euler3d": (dgp.LAW_EULER3D, dgp.FLUX_GODUNOV, dgp.FIELD_PULSE3D, PULSE3D),
            "euler": (dgp.LAW_EULER2D, dgp.FLUX_ROE, dgp.FIELD_VORTEX, VORTEX)}[kind]
    s = dgp.Solver(_mesh(3 if kind.endswith("3d") else 2, 4, 3, box=10.0), dgp.Law(*args), order)
    s.set_fused(False)
    assert s.block() == (128, elem)
    u0 = s.get_state()
    t, n = s.run(0.0, 0.0, 0.1, 3)
    u = s.get_state()
    s.set_fused(True)
    assert s.block() == (128, stage)
    s.set_state(u0)
    assert s.run(0.0, 0.0, 0.1, 3)[1] == n == 3
    assert rel(s.get_state(), u) < 1e-12


# the default form at sizes where the other one was measured slower or faster
@pytest.mark.parametrize("kind,order,precision,n,fused", [
    ("scalar3d", 3, dgp.FP64, 4, False), ("scalar3d", 3, dgp.MIXED, 15, True), ("scalar3d", 2, dgp.FP64, 4, True),
    ("maxwell3d", 3, dgp.FP64, 4, False), ("maxwell3d", 3, dgp.MIXED, 4, False), ("maxwell3d", 3, dgp.MIXED, 10, True),
    ("euler3d", 1, dgp.FP64, 4, False), ("euler3d", 1, dgp.MIXED, 4, True), ("euler3d", 3, dgp.MIXED, 10, False),
    ("euler", 4, dgp.FP64, 20, False), ("euler", 4, dgp.FP64, 60, True), ("euler", 3, dgp.FP64, 20, True),
    ("euler", 0, dgp.FP64, 20, True), ("euler", 0, dgp.FP64, 210, False), ("scalar", 4, dgp.FP64, 20, True)])
def test_default_form(kind, order, precision, n, fused):
    args = {"scalar3d": (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS3D, SCALAR3D),
            "scalar": (dgp.LAW_SCALAR, dgp.FLUX_UPWIND, dgp.FIELD_GAUSS, SCALAR2D),
            "maxwell3d": (dgp.LAW_MAXWELL3D, dgp.FLUX_UPWIND, dgp.FIELD_TM110, TM110),
            "euler3d": (dgp.LAW_EULER3D, dgp.FLUX_GODUNOV, dgp.FIELD_PULSE3D, PULSE3D),
            "euler": (dgp.LAW_EULER2D, dgp.FLUX_ROE, dgp.FIELD_VORTEX, VORTEX)}[kind]
    s = dgp.Solver(_mesh(3 if kind.endswith("3d") else 2, n, 3, box=10.0), dgp.Law(*args), order, precision)
    assert s.fused == fused


# an ensemble of each form whose tiles differ (17 / 25 cells, 14 / 21), in FP64
@pytest.mark.parametrize("kind", ["euler3d", "maxwell3d"])
def test_ensembles_start_instances_on_their_forms_tiles(kind):
    args = (dgp.LAW_EULER3D, dgp.FLUX_GODUNOV, dgp.FIELD_PULSE3D, PULSE3D) if kind == "euler3d" else \
        (dgp.LAW_MAXWELL3D, dgp.FLUX_UPWIND, dgp.FIELD_TM110, TM110)
    tag = 40000 if kind == "maxwell3d" else 1
    meshes = [_mesh(3, n, n, tag) for n in (2, 4, 3)]
    laws = [dgp.Law(*args) for _ in meshes]
    e = dgp.Ensemble(meshes, laws, [2, 2, 2])
    assert e.group_block(0) == (128, 17 if kind == "euler3d" else 21)
    e.project(0.0)
    t, n, _, _ = e.run(0.0, 0.0, 0.1, 5)
    for i in range(3):
        s = dgp.Solver(meshes[i], laws[i], 2)
        assert s.fused == (kind == "maxwell3d")
        s.project(0.0)
        ts, ns = s.run(0.0, 0.0, 0.1, 5)
        assert n[i] == ns == 5 and abs(t[i] - ts) <= 1e-14 * ts
        assert np.array_equal(e.get_state(i), s.get_state())


def test_autotune_times_both_forms_of_an_ensemble():
    meshes = [_mesh(2, n, n) for n in (15, 16)]
    laws = [dgp.Law(dgp.LAW_BURGERS2D, dgp.FLUX_LLF, dgp.FIELD_SINE, SINE) for _ in meshes]
    dgp.autotune_ensemble(meshes, laws, [4, 4], dgp.FP64, iters=2)
    e = dgp.Ensemble(meshes, laws, [4, 4])
    e.project(0.0)
    e.run(0.0, 0.0, 0.1, 4)
    for i in range(2):
        s = dgp.Solver(meshes[i], laws[i], 4)
        s.project(0.0)
        s.run(0.0, 0.0, 0.1, 4)
        assert rel(e.get_state(i), s.get_state()) < 1e-13


def test_default_form_gives_way_where_only_the_fused_one_can():
    """The separate kernels as a default, not as the caller's choice, refuse
    nothing: the tensor cores switch to the fused form, and a right-hand side
    without allocations takes it (145800 cells need 36 MiB of slots otherwise)."""
    args = (dgp.LAW_EULER3D, dgp.FLUX_GODUNOV, dgp.FIELD_PULSE3D, PULSE3D)
    s, c = (dgp.Solver(_mesh(3, 4, 3), dgp.Law(*args), 2, dgp.MIXED) for _ in range(2))
    assert not s.fused
    s.set_tensor_cores(True)
    assert s.fused
    s.run(0.0, 0.0, 0.1, 2)
    c.set_fused(False)
    with pytest.raises(dgp.DGPError):
        c.set_tensor_cores(True)
    c.run(0.0, 0.0, 0.1, 2)
    assert rel(s.get_state(), c.get_state()) < 2e-5

    torch = pytest.importorskip("torch")
    s = dgp.Solver(_mesh(2, 270, 3, box=10.0), dgp.Law(dgp.LAW_EULER2D, dgp.FLUX_ROE, dgp.FIELD_VORTEX, VORTEX), 0)
    assert not s.fused
    u = torch.from_numpy(s.get_state().ravel().copy()).cuda()
    r = torch.full_like(u, float("nan"))
    torch.cuda.synchronize()
    assert rhs_noalloc(s, u.data_ptr(), 0.2, r.data_ptr()) == 0
    assert rel(r.cpu().numpy().reshape(s.shape), s.rhs(0.2)) < 1e-12
