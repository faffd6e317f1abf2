"""The Hex27 sweep at the edges of its 32-element tiles, in each geometry form, phase layout and
number of phases, with every optional field, against the oracle."""
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


def off_alignment(x):
    """The same values at an address that is a multiple of the entry's size only."""
    buf = torch.empty(x.numel() + 1, dtype=x.dtype, device=x.device)
    return buf[1:].view(x.shape).copy_(x)


# n³ elements: one, a part of a tile, two whole tiles, three and a part, seven tiles less nine
# elements. An entry sums 27 points × 27 nodes of terms below ~100 times its scale: 1e4 units in the
# last place; a float geometry alone brings 6e-8 of each term.
@pytest.mark.parametrize("dtypes,rtol", [(("f64", "f64"), 1e-11), (("f32", "f32"), 2e-3), (("f64", "f32"), 2e-5)])
@pytest.mark.parametrize("n,cells,phases,nph,fields", [
    (1, "points", "nodal", 3, "none"), (3, "points", "element", 4, "all"), (4, "sheared", "nodal", 2, "all"),
    (5, "box", "element", 6, "P_old"), (5, "points", "nodal", 6, "eta"), (6, "sheared", "cell", 3, "all"),
    (6, "box", "cell", 3, "none"), (5, "points", "cell", 3, "all"), (3, "box", "nodal", 4, "unaligned"),
    (4, "points", "cell", 2, "unaligned")])
def test_hex27_edges(n, cells, phases, nph, fields, dtypes, rtol):
    case = random_state_case(dim=3, n=n, seed=60 + n, phases=phases, nphases=nph, distort=cells == "points")
    mesh = case.mesh
    rng = np.random.default_rng(n)
    if cells == "box":
        c = mesh.coords
        c[:, 1] -= 0.1 * c[:, 2]
        c[:, 0] -= 0.2 * c[:, 1]
        mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    # contrasts that keep the quadratic interpolation of mixed phases positive (a pole otherwise)
    u = lambda lo, hi: tuple(rng.uniform(lo, hi, nph))
    case.material = fem.StokesMaterial(eta=u(1, 2), eta_b=u(15, 30), G=u(1, 2), alpha=u(.05, .1), rho0=u(1, 2), K=u(40, 80),
                                       g=(0.1, 0.3, -1.0), Tref=0.1)
    case.plastic = fem.DruckerPrager.from_angles(u(.3, .6), u(.1, .2), u(.15, .3), u(.05, .1), u(5, 10))
    td, gd = (torch.float64 if d == "f64" else torch.float32 for d in dtypes)
    dr, hs = case.device_state(fem, dtype=td, geometry_dtype=gd), case.host_state(oh)
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
    if fields == "unaligned":
        dr._mesh["geo_v"] = off_alignment(dr._mesh["geo_v"])
        for c in (0, 4):
            dr.tau_old[c] = off_alignment(dr.tau_old[c])
    fem.assemble_stokes_residuals(dr, case.dt)
    hs.stokes_residuals(case.dt)
    near(dr.RP, hs.RP, rtol, "RP")
    near(dr.Pnum, hs.Pnum, rtol, "Pnum")
    for c in range(3):
        near(dr.Rv[c], hs.Rv[c], rtol, f"Rv[{c}]")
    near(fem.assemble_shear_heating(dr, case.dt), hs.shear_heating(case.dt), rtol, "phi")
    for with_pnum in (False, True):   # stored Pnum, pressure pass off
        dr.Pnum.copy_(dev(case.Pnum)); hs.Pnum[:] = case.Pnum
        fem.assemble_momentum_residual(dr, case.dt, with_pnum=with_pnum)
        hs.momentum_residual(case.dt, with_pnum=with_pnum)
        for c in range(3):
            near(dr.Rv[c], hs.Rv[c], rtol, f"Rv[{c}] stored Pnum")
    dr.viscosity_ip = None
    hs.viscosity_ip = None
    fem.update_stokes_current_stress(dr, case.dt)
    hs.store_stress(case.dt)
    for c in range(6):
        near(dr.tau[c], hs.tau[c], rtol, f"tau[{c}]")
