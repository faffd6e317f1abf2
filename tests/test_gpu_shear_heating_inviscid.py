"""Shear heating where a phase, or some integration points, have no viscosity: no stress, so no
heating, as the oracle gives it."""
import numpy as np
import pytest

import oracle_host as oh
from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# a point's heating is a few products of the stress and the gradient, each below their scale
# by no more than 100 units in the last place
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("field", [False, True])
def test_no_viscosity(dim, field):
    case = random_state_case(dim=dim, n=3, seed=4, phases="cell", plastic=False, distort=dim == 3)
    m = case.material
    if not field:
        case.material = fem.StokesMaterial(eta=(0.0,) + tuple(m.eta[1:]), eta_b=m.eta_b, G=m.G, alpha=m.alpha, rho0=m.rho0,
                                           K=m.K, g=m.g, Tref=m.Tref)
    dr, hs = case.device_state(fem), case.host_state(oh)
    none = np.repeat(case.phases_v == 1, case.mesh.nq)
    if field:
        hs.viscosity_ip = np.where(none, 0.0, np.random.default_rng(1).uniform(1, 2, none.size))
        dr.viscosity_ip = dr.tensor(hs.viscosity_ip)
    got = fem.assemble_shear_heating(dr, case.dt).cpu().numpy()
    want = hs.shear_heating(case.dt)
    assert none.any() and (want[none] == 0).all() and (got[none] == 0).all()
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
