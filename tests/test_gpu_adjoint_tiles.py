"""One iteration of the adjoint solve, whose operator comes from the frozen state's pull-back
coefficients, against the operator formed anew: partial and several tiles, per-point and affine
geometry, every phase layout, without plasticity, with a viscosity field and a fluid pressure."""
import numpy as np
import pytest

from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cells,phases,plastic,eta,finite_K", [
    (1, "distorted", "nodal", True, False, False), (3, "distorted", "element", True, True, True),
    (4, "sheared", "cell", True, False, False), (5, "sheared", "nodal", False, True, False),
    (6, "distorted", "cell", True, False, True), (18, "sheared", "cell", True, False, False)])
def test_frozen_operator(n, cells, phases, plastic, eta, finite_K):
    case = random_state_case(dim=3, n=n, seed=70 + n, phases=phases, plastic=plastic, distort=cells == "distorted")
    rng = np.random.default_rng(n)
    u = lambda lo, hi: tuple(rng.uniform(lo, hi, 3))
    # contrasts that keep the quadratic interpolation of mixed phases positive (a pole otherwise)
    case.material = fem.StokesMaterial(eta=u(1, 2), eta_b=u(15, 30), G=u(1, 2), alpha=u(.05, .1), rho0=u(1, 2), K=u(40, 80),
                                       g=(0.1, 0.3, -1.0), Tref=0.1)
    if plastic:
        case.plastic = fem.DruckerPrager.from_angles(u(.3, .6), u(.1, .2), u(.15, .3), u(.05, .1), u(5, 10))
    dr = case.device_state(fem)
    mesh = case.mesh
    rand = lambda k: dr.tensor(rng.standard_normal(k))
    if eta:
        dr.viscosity_ip = dr.tensor(rng.uniform(1, 2, mesh.nq * mesh.nels))
        dr.Pf.copy_(0.1 * rand(mesh.nnodesP))
        dr._use_Pf = True
    lv, lP, obj = [rand(mesh.nnodes) for _ in range(3)], rand(mesh.nnodesP), [rand(mesh.nnodes) for _ in range(3)]
    b = mesh.boundary_nodes[:5]
    bc = [fem.DirichletBoundaryCondition(b, np.zeros(len(b)))] * 3
    for c in range(3):
        lv[c][torch.as_tensor(b - 1, device="cuda").long()] = 0.0
    v0, P0 = [x.clone() for x in lv], lP.clone()
    ref_v, _ = fem.assemble_adjoint_residual(dr, case.dt, v0, P0, finite_K=finite_K)
    _, _, st = fem.solve_adjoint(dr, bc, case.dt, obj, lam_v=lv, lam_P=lP, max_iterations=1, max_ph_iterations=1,
                                 tolerance=1e-300, throw_on_failure=False, finite_K=finite_K)
    assert st["iter"] == 1
    _, ref_P = fem.assemble_adjoint_residual(dr, case.dt, lv, P0, finite_K=finite_K)
    # λP += γP·ResP/M_P at the updated λv; λv −= α·Resv/PC with one α per component. An entry sums 27
    # points of 27 nodes' terms below ~100 times its scale (1e4 units in the last place); the
    # differences below lose no more than the ratio of λ to its step, under 10
    near = lambda x, y: float((x - y).abs().max()) <= 1e-11 * float(y.abs().max())
    assert near((lP - P0) * dr.M_P / dr.gammaP, ref_P)
    free = torch.ones(mesh.nnodes, dtype=torch.bool, device="cuda")
    free[torch.as_tensor(b - 1, device="cuda").long()] = False
    for c in range(3):
        step = (ref_v[c] + obj[c]) / dr.PC[c]
        d = (v0[c] - lv[c])[free]
        alpha = float(d @ step[free]) / float(step[free] @ step[free])
        assert alpha > 0 and not (lv[c][~free] != 0).any()
        assert near(v0[c][free] - alpha * step[free], lv[c][free])
