"""The adjoint solve's table of pull-back coefficients: what a solve holds on to, and the solve
without it (what one without the memory for it does)."""
import ctypes as C
import os

import numpy as np
import pytest

from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi


def handle(monkeypatch, table=True):
    """A handle of its own, in the place of the process's."""
    if not table:
        monkeypatch.setenv("FEMB200_ADJOINT_TABLE", "0")
    h = C.c_void_p()
    assert abi.load_library().femb200_create(C.byref(h)) == abi.OK
    monkeypatch.setattr(fem.solver._Handle, "_h", h)
    return h


# a residual entry sums 27 points' terms of 27 nodes below ~100 times its scale (1e4 units in the last
# place); three Chebyshev steps carry the differences on
@pytest.mark.parametrize("n,cells,phases,plastic", [(3, "distorted", "nodal", True), (4, "sheared", "cell", True),
                                                    (4, "sheared", "cell", False)])
def test_without_the_table(monkeypatch, n, cells, phases, plastic):
    case = random_state_case(dim=3, n=n, seed=90 + n, phases=phases, plastic=plastic, distort=cells == "distorted")
    case.material = fem.StokesMaterial(eta=(1.0, 1.5, 2.0), eta_b=(20.0,) * 3, G=(1.0, 1.5, 2.0), alpha=(0.1,) * 3,
                                       rho0=(1.0, 1.5, 2.0), K=(50.0, 60.0, 70.0), g=(0.1, 0.3, -1.0), Tref=0.1)
    rng = np.random.default_rng(n)
    b = case.mesh.boundary_nodes
    bc = [fem.DirichletBoundaryCondition(b, np.zeros(len(b)))] * 3
    obj = [rng.standard_normal(case.mesh.nnodes) for _ in range(3)]
    out = []
    for table in (True, False):
        with monkeypatch.context() as m:
            h = handle(m, table)
            dr = case.device_state(fem)
            lv, lP, st = fem.solve_adjoint(dr, bc, case.dt, [dr.tensor(o) for o in obj], max_iterations=3, iter_max=3,
                                           tolerance=1e-300, throw_on_failure=False)
            torch.cuda.synchronize()
            abi.load_library().femb200_destroy(h)
        out.append([*lv, lP])
    for got, want in zip(*out):
        assert float(want.abs().max()) > 0
        assert float((got - want).abs().max()) <= 1e-10 * float(want.abs().max())


@pytest.mark.parametrize("plastic", [True, False])
def test_a_large_table_is_given_back(monkeypatch, plastic):
    nel = (48, 48, 48)
    el2n = fem.mesh.structured_connectivity(3, nel)
    ax = [np.linspace(0, 1, 2 * k + 1) for k in nel]
    z, y, x = np.meshgrid(*ax[::-1], indexing="ij")
    coords = np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1)
    geo_v, geo_P = fem.precompute_geometry(coords, el2n, 3)
    nels = len(el2n)
    dofs = (np.arange(4 * nels, dtype=np.int32) + 1).reshape(nels, 4)
    mesh = fem.MixedMesh(3, nel, coords, el2n, dofs, el2n[:, [26, 22, 23, 25]].copy(), geo_v, geo_P, np.array([1], dtype=np.int32))
    mat = fem.StokesMaterial(eta=(1.0,), eta_b=(10.0,), G=(1.0,), alpha=(0.0,), rho0=(1.0,), K=(10.0,), g=(0.0, 0.0, -1.0))
    pl = fem.DruckerPrager.from_angles((0.5,), (0.0,), (0.3,), (0.1,), (10.0,)) if plastic else None
    dr = fem.StokesDR(mesh, mat, pl)
    fem.assemble_viscosity_weighted_pressure_scaling(dr, 50.0, 1.0)
    bc = [fem.DirichletBoundaryCondition(np.array([1], dtype=np.int32), np.zeros(1))] * 3
    one = lambda n: torch.ones(n, dtype=torch.float64, device="cuda")
    lv, lP, obj = [one(mesh.nnodes) for _ in range(3)], one(mesh.nnodesP), [one(mesh.nnodes) for _ in range(3)]
    h = handle(monkeypatch)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    fem.solve_adjoint(dr, bc, 1.0, obj, lam_v=lv, lam_P=lP, max_iterations=1, iter_max=1, tolerance=1e-300, throw_on_failure=False)
    held = before - torch.cuda.mem_get_info()[0]
    abi.load_library().femb200_destroy(h)
    # the iteration's vectors, the compressed geometry and masks; no table above 256 MB (287 MB here with
    # plasticity, 72 without, where twelve fields a point would be 287)
    rest = 8 * (9 * mesh.nnodes + mesh.nnodesP) + 80 * nels + mesh.nnodes
    assert held <= rest + (0 if plastic else 8 * 3 * 27 * nels) + (32 << 20)
