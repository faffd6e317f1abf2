"""FP64 Jacobian diagnostics on axis-aligned boxes: elastic tiles, tiles with yielding points and
meshes with both, one and several tiles, against the oracle."""
import numpy as np
import pytest

import oracle_host as oh
from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# n³ elements: one, a part of a tile, two whole tiles, seven less nine elements. A row sum adds 81
# entries of 27 points' terms, all at most of its own scale: 2 187 units in the last place, 5e-13;
# the geometry of a cell agrees with its centre's to 1e-12
@pytest.mark.parametrize("n,state", [(1, "elastic"), (1, "yield"), (3, "elastic"), (4, "yield"), (4, "viscous"), (6, "mixed"),
                                     (6, "elastic")])
@pytest.mark.parametrize("field", [False, True])
def test_jacobian_box(n, state, field):
    case = random_state_case(dim=3, n=n, seed=80 + n, phases="cell", plastic=state != "viscous", distort=False)
    mesh, rng = case.mesh, np.random.default_rng(n)
    c = mesh.coords
    c[:, 1] -= 0.1 * c[:, 2]
    c[:, 0] -= 0.2 * c[:, 1]
    c *= (1.0, 0.7, 1.3)
    mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    if state in ("elastic", "mixed"):
        # far below yield; in the second half of the elements of `mixed` as drawn
        low = 1e-3 if state == "elastic" else np.where(np.arange(mesh.nels) < mesh.nels // 2, 1e-3, 1.0)
        for k in range(3):
            x = 1e-3 * case.v[k]
            case.v[k][:] = x
        for k in range(6):
            case.tau_old[k] = (case.tau_old[k].reshape(mesh.nels, -1) * np.reshape(low, (-1, 1))).ravel()
        case.P = 1.0 + 1e-3 * case.P if state == "elastic" else case.P
    dr, hs = case.device_state(fem), case.host_state(oh)
    if field:
        hs.viscosity_ip = rng.uniform(1, 2, mesh.nq * mesh.nels)
        dr.viscosity_ip = dr.tensor(hs.viscosity_ip)
        hs.Pf[:] = 0.1 * rng.standard_normal(mesh.nnodesP)
        dr.Pf.copy_(dr.tensor(hs.Pf))
        dr._use_Pf = True
    fem.assemble_augmented_momentum_jacobian(dr, case.dt)
    hs.jacobian_diagnostics(case.dt)
    for k in range(3):
        for got, want in ((dr.dRdv[k], hs.dRdv[k]), (dr.PC[k], hs.PC[k])):
            assert np.abs(got.cpu().numpy() - want).max() <= 5e-12 * np.abs(want).max()
