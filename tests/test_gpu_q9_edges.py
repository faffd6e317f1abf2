"""The Q9 sweep and Jacobian diagnostics at the edges of their 32-element tiles and
three-element groups, with every optional field, against the oracle."""
import numpy as np
import pytest

import oracle_host as oh
from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi


def near(got, ref, rtol, what):
    ref = np.asarray(ref)
    assert np.abs(got.double().cpu().numpy() - ref).max() <= rtol * max(np.abs(ref).max(), 1e-300), what


# n² elements: one, a part of a tile, a tile and a part, two tiles
# (an entry sums 9 points × 9 nodes of terms below ~100 times its scale: 1e4 units in the last place)
@pytest.mark.parametrize("dtype,rtol", [("f64", 1e-11), ("f32", 2e-3)])
@pytest.mark.parametrize("n,phases,fields", [(1, "nodal", "none"), (5, "cell", "all"), (6, "element", "P_old"),
                                             (6, "cell", "eta"), (8, "nodal", "all"), (6, "cell", "none")])
def test_q9_edges(n, phases, fields, dtype, rtol):
    case = random_state_case(dim=2, n=n, seed=40 + n, phases=phases)
    # contrasts that keep the quadratic interpolation of mixed phases positive (a pole otherwise)
    rng = np.random.default_rng(n)
    u = lambda lo, hi: tuple(rng.uniform(lo, hi, 3))
    case.material = fem.StokesMaterial(eta=u(1, 2), eta_b=u(15, 30), G=u(1, 2), alpha=u(.05, .1), rho0=u(1, 2), K=u(40, 80),
                                       g=(0.1, -1.0), Tref=0.1)
    case.plastic = fem.DruckerPrager.from_angles(u(.3, .6), u(.1, .2), u(.15, .3), u(.05, .1), u(5, 10))
    td = torch.float64 if dtype == "f64" else torch.float32
    dr, hs = case.device_state(fem, dtype=td, geometry_dtype=td), case.host_state(oh)
    mesh = case.mesh
    dev = lambda x: torch.as_tensor(x, dtype=td, device="cuda")
    if fields in ("all", "eta"):
        hs.viscosity_ip = rng.uniform(1, 2, mesh.nq * mesh.nels)
        dr.viscosity_ip = dev(hs.viscosity_ip)
    if fields in ("all", "P_old"):
        hs.P_old, hs.P_old_layout = rng.standard_normal(mesh.nq * mesh.nels), abi.FIELD_IP
        dr.P_old, dr.P_old_layout = dev(hs.P_old), abi.FIELD_IP
    if fields == "all":
        for name in ("Q", "Pf"):
            x = 0.1 * rng.standard_normal(mesh.nnodesP)
            getattr(hs, name)[:] = x
            getattr(dr, name).copy_(dev(x))
        dr._use_Q = dr._use_Pf = True
    fem.assemble_stokes_residuals(dr, case.dt)
    hs.stokes_residuals(case.dt)
    near(dr.RP, hs.RP, rtol, "RP")
    near(dr.Pnum, hs.Pnum, rtol, "Pnum")
    for c in range(2):
        near(dr.Rv[c], hs.Rv[c], rtol, f"Rv[{c}]")
    near(fem.assemble_shear_heating(dr, case.dt), hs.shear_heating(case.dt), rtol, "phi")
    fem.assemble_augmented_momentum_jacobian(dr, case.dt)
    hs.jacobian_diagnostics(case.dt)
    for c in range(2):
        near(dr.dRdv[c], hs.dRdv[c], rtol, f"dRdv[{c}]")
        near(dr.PC[c], hs.PC[c], rtol, f"PC[{c}]")
    for with_pnum in (False, True):   # stored Pnum, pressure pass off
        dr.Pnum.copy_(dev(case.Pnum)); hs.Pnum[:] = case.Pnum
        fem.assemble_momentum_residual(dr, case.dt, with_pnum=with_pnum)
        hs.momentum_residual(case.dt, with_pnum=with_pnum)
        for c in range(2):
            near(dr.Rv[c], hs.Rv[c], rtol, f"Rv[{c}] stored Pnum")
    dr.viscosity_ip = None
    hs.viscosity_ip = None
    fem.update_stokes_current_stress(dr, case.dt)
    hs.store_stress(case.dt)
    for c in range(3):
        near(dr.tau[c], hs.tau[c], rtol, f"tau[{c}]")
