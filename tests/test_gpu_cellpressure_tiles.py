"""Iterations of the cell-pressure relaxation on one and several tiles of 32 elements, affine and
distorted cells, against the oracle: free walls (the mean of the constant pressure mode then acts on
the wall nodes), with a check in between."""
import numpy as np
import pytest

import oracle_host as oh
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# a tile holds 32 elements; 18³ are more tiles than multiprocessors. An entry after three iterations
# sums three times 27 points of 27 nodes' terms below ~100 times its scale: 1e4 units in the last place
@pytest.mark.parametrize("n,distort", [(1, True), (1, False), (4, False), (5, True), (18, False), (6, True)])
def test_iterations(n, distort):
    case = fem.configs.cell_pressure_case(n=n, seed=n, distort=distort)
    rng = np.random.default_rng(n)
    v = [rng.standard_normal(case.mesh.nnodes) for _ in range(3)]
    P = 1.0 + rng.standard_normal(4 * case.mesh.nels)
    bc = [case.bc[0], (case.bc[1][0][:3], np.array([0.1, -0.2, 0.3])), (np.zeros(0, np.int32), np.zeros(0))]
    dr = fem.CellPressureStokesDR(case.mesh, case.material, phases=case.phases)
    for c in range(3):
        dr.v[c].copy_(torch.as_tensor(v[c], device="cuda"))
    dr.P.copy_(torch.as_tensor(P, device="cuda"))
    hs = oh.HostCellPressure(case.mesh, case.material.eta, case.material.rho0, case.material.g, case.phases, v, P)
    kw = dict(tolerance=1e-30, max_iterations=3, check_interval=2)
    st = fem.solve_cell_pressure(dr, bc, throw_on_failure=False, **kw)
    ref = hs.solve(bc, throw_on_failure=False, **kw)
    assert st["iterations"] == ref.iterations == 3
    for got, want in zip([*dr.v, dr.P, dr.RP, *dr.Rv], [*hs.v, hs.P, hs.RP, *hs.Rv]):
        assert np.abs(got.cpu().numpy() - want).max() <= 1e-11 * max(np.abs(want).max(), 1e-300)
    assert abs(st["residual"] - ref.residual) <= 1e-11 * ref.residual
