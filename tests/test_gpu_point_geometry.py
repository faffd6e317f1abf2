"""Cells whose integration points carry slightly different geometry: every point's J⁻¹ and weight is
scaled by 1 + 9e-13 except the centre's, less than the 1e-12 to which the affine sweeps let a cell's
points differ. What reads the geometry per point must show the difference as a common factor of its result."""
import numpy as np
import pytest

import oracle_host as oh
from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DELTA = 9e-13
# A common factor of 1 + 9e-13 in J⁻¹ and the weights changes a flux integral by 2.7e-12, a value integral
# by 9e-13. The roundings of the ~1 000 entries projected on are independent and below 100
# units in the last place of their scale: 4e-16 in the projection
LIMIT = 1e-13


def scaled(mesh):
    f = np.full(27, 1.0 + DELTA)
    f[13] = 1.0
    mesh.geo_v, mesh.geo_P = mesh.geo_v * f[None, :, None], mesh.geo_P * f[None, :]
    return mesh


def off16(x):
    """A copy eight bytes off a 16-byte boundary."""
    y = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)[1:].view(x.shape)
    return y.copy_(x)


def factor(got, want):
    """Relative difference of two arrays along the second."""
    got, want = (np.asarray(x.cpu() if hasattr(x, "cpu") else x, dtype=np.float64) for x in (got, want))
    return abs((got - want) @ want) / (want @ want)


@pytest.mark.parametrize("nel,sheared,aligned", [((5, 4, 3), False, True), ((9, 3, 4), True, True), ((5, 4, 3), True, False)])
def test_thermal_solve(nel, sheared, aligned):
    rng = np.random.default_rng(sum(nel))
    mesh = fem.structured_mixed_mesh(3, nel)
    if sheared:
        c = mesh.coords
        c[:, 0] += 0.2 * c[:, 1]
        mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    scaled(mesh)
    kw = dict(k=(1.0,), Cp=(1.3,), rho0=(1.2,), alpha=(0.05,), K=(50.0,))
    th, ht = fem.ThermalDiffusionDR(mesh, **kw), oh.HostThermal(mesh, **kw)
    if not aligned:
        th.geo = off16(th.geo)
    for name in ("T", "T0", "source", "P"):
        x = rng.uniform(0, 1, mesh.nnodes)
        getattr(th, name).copy_(torch.as_tensor(x))
        getattr(ht, name)[:] = x
    dofs, vals = mesh.boundary_nodes[:3], np.array([0.2, 0.4, 0.6])
    ht.set_bc(dofs, vals)
    run = dict(dt=0.1, Tref=0.3, tolerance=1e-300, max_iterations=3, check_interval=4, throw_on_failure=False)
    fem.solve_thermal(th, fem.DirichletBoundaryCondition(dofs, vals), **run)   # iterations 2 and 3: no Jacobian
    ht.solve(**run)
    assert factor(th.R, ht.R) <= LIMIT


@pytest.mark.parametrize("aligned", [True, False])
def test_adjoint_solve(aligned):
    n = 5
    case = random_state_case(dim=3, n=n, seed=11, phases="cell", plastic=False, nphases=1, distort=False)
    mesh = scaled(case.mesh)
    rng = np.random.default_rng(n)
    dr = case.device_state(fem)
    if not aligned:
        dr._mesh["geo_v"] = off16(dr._mesh["geo_v"])
    rand = lambda k: dr.tensor(rng.standard_normal(k))
    lv, lP, obj = [rand(mesh.nnodes) for _ in range(3)], rand(mesh.nnodesP), [rand(mesh.nnodes) for _ in range(3)]
    b = mesh.boundary_nodes[:5]
    bc = [fem.DirichletBoundaryCondition(b, np.zeros(len(b)))] * 3
    P0 = lP.clone()
    _, _, st = fem.solve_adjoint(dr, bc, case.dt, obj, lam_v=lv, lam_P=lP, max_iterations=1, max_ph_iterations=1,
                                 tolerance=1e-300, throw_on_failure=False)
    assert st["iter"] == 1
    # λP += γP·ResP/M_P with the operator of the iteration, at the updated λv
    _, ref_P = fem.assemble_adjoint_residual(dr, case.dt, lv, P0)
    assert factor((lP - P0) * dr.M_P / dr.gammaP, ref_P) <= LIMIT


def test_coupled_shear_heating():
    n = 5
    case = random_state_case(dim=3, n=n, seed=12, phases="cell", plastic=False, nphases=1, distort=False)
    mesh = scaled(case.mesh)
    dr = case.device_state(fem)
    th = fem.ThermalDiffusionDR(mesh, k=(1.0,), Cp=(1.3,), rho0=(1.2,))
    bc_T = fem.DirichletBoundaryCondition(mesh.boundary_nodes[:3], np.zeros(3))
    bc_v = [fem.DirichletBoundaryCondition(mesh.boundary_nodes[:5], np.zeros(5))] * 3
    ref = fem.assemble_shear_heating(dr, case.dt).clone()
    # the first iteration's heating is that of the velocities before their first update
    _, phi = fem.solve_coupled(th, dr, bc_T, bc_v, case.dt, Tref=0.1, shear_heating=True, max_iterations=0, throw_on_failure=False)
    assert factor(phi, ref) <= LIMIT


def test_small_off_diagonal_entries():
    """A J⁻¹ with one off-diagonal entry of 8e-15 of its diagonal, and a velocity whose divergence is that
    entry times its gradient: v_x = y on a box."""
    mesh = fem.structured_mixed_mesh(3, (4, 4, 4))
    mesh.geo_v[:, :, 1] = 8e-15 * mesh.geo_v[:, :, 0]   # ∂η/∂x
    mat = fem.StokesMaterial(eta=(1.0,), eta_b=(np.inf,), G=(np.inf,), alpha=(0.0,), rho0=(0.0,), K=(np.inf,), g=(0.0, 0.0, 0.0))
    dr = fem.StokesDR(mesh, mat, None)
    dr.v[0].copy_(dr.tensor(mesh.coords[:, 1]))
    fem.assemble_pressure_residual(dr, 1.0)
    # RP_0 = −Σ_q N_0 ∂η/∂x ∂v_x/∂η dΩ with ∂v_x/∂η = h/2 = 1/8, ∂ξ/∂x = 8 and Σ_q N_0 dΩ = 1/64. The
    # rounding of the other terms is that of ∂v_x/∂ξ, zero on a line of equal values
    want = -8e-15 / 64
    got = dr.RP.cpu().numpy()[::4]
    assert np.abs(got - want).max() <= 0.2 * abs(want)


# elastic: closed form per cell; yielding: 81 columns; both only where a cell's points agree to rounding.
# Row sums of absolute values add up no cancelling roundings: their common factor is known better still
@pytest.mark.parametrize("plastic", [False, True])
def test_jacobian(plastic):
    case = random_state_case(dim=3, n=5, seed=13, phases="cell", plastic=plastic, distort=False)
    mesh = case.mesh
    c = mesh.coords
    c[:, 1] -= 0.1 * c[:, 2]
    c[:, 0] -= 0.2 * c[:, 1]
    mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    mesh.geo_v[..., [1, 2, 3, 5, 6, 7]] = 0.0
    scaled(mesh)
    dr, hs = case.device_state(fem), case.host_state(oh)
    fem.assemble_augmented_momentum_jacobian(dr, case.dt)
    hs.jacobian_diagnostics(case.dt)
    for k in range(3):
        assert factor(dr.dRdv[k], hs.dRdv[k]) <= LIMIT
        assert factor(dr.PC[k], hs.PC[k]) <= LIMIT
