"""A Stokes problem without a temperature but with an earlier one: the absent field is zero."""
import pytest

from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,distort", [(2, True), (3, False), (3, True)])
def test_absent_temperature(dim, distort):
    case = random_state_case(dim=dim, n=3, seed=6, phases="cell", plastic=True, distort=distort)
    dr = case.device_state(fem)
    dr.T.zero_()
    fem.assemble_stokes_residuals(dr, case.dt)
    want = [x.clone() for x in (dr.RP, *dr.Rv)]
    dr.T0.zero_()
    fem.assemble_pressure_residual(dr, case.dt)
    assert float((dr.RP - want[0]).abs().max()) > 1e-3 * float(want[0].abs().max())   # T0 counts
    dr.T0.copy_(dr.tensor(case.T0))
    dr.T = None
    fem.assemble_stokes_residuals(dr, case.dt)
    # the pressure residual is the same sum; the nodal ones add in another order (8 elements an entry)
    assert torch.equal(dr.RP, want[0])
    for got, w in zip(dr.Rv, want[1:]):
        assert float((got - w).abs().max()) <= 1e-14 * float(w.abs().max())
