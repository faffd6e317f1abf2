"""The tiled FP32 incremental sweep against the FP64 sweep over a few iterations of the same
solve: partial and single-element tiles, tiles that cross rows, full J⁻¹, yielding points, and base
states at the yield-surface apex (their tiles take the FP64 return)."""
import math

import numpy as np
import pytest

from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi


def state(nel, seed, shear, load):
    rng = np.random.default_rng(seed)
    mesh = fem.structured_mixed_mesh(3, nel)
    c = mesh.coords
    if shear:
        c[:, 0] += 0.2 * c[:, 1]
        c[:, 1] += 0.1 * c[:, 2]
        mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    ph = rng.integers(1, 3, mesh.nels).astype(np.int32)
    mat = fem.StokesMaterial(eta=(1.0, 10.0), eta_b=(10.0,) * 2, G=(1.0,) * 2, alpha=(0.0,) * 2, rho0=(1.0, 1.5),
                             K=(10.0,) * 2, g=(0.1, 0.2, -1.0))
    pl = fem.DruckerPrager.from_angles((math.radians(30),) * 2, (0.0,) * 2, (0.3, 0.5), (0.1,) * 2, (10.0,) * 2)
    dr = fem.StokesDR(mesh, mat, pl, phases_v=ph, phases_v_layout=abi.PHASE_CELL, phases_P=ph, phases_P_layout=abi.PHASE_CELL)
    f = [c[:, 0] - 0.5, np.zeros(mesh.nnodes), -(c[:, 2] - 0.5)] if load != "apex" else [np.zeros(mesh.nnodes)] * 3
    dr.set_velocity(f)
    n = mesh.nq * mesh.nels
    if load == "yield":
        t = 0.3 * (1 + 0.2 * rng.standard_normal(n))
        dr.tau_old[0].copy_(dr.tensor(t)); dr.tau_old[2].copy_(dr.tensor(-t))
        dr.tau_old[3].copy_(dr.tensor(0.05 * rng.standard_normal(n)))
    if load == "apex":
        # a little below yield at the apex pressure −C·cotϕ, with no deviatoric stress in two
        # thirds of the points
        C = np.array([0.3, 0.5])[ph - 1]
        dr.P.copy_(dr.tensor(np.repeat(-(C * math.cos(math.radians(30)) - 1e-3) / 0.5, 4)))
        dr.tau_old[0].copy_(dr.tensor(np.where(np.arange(n) % 3 == 0, 2e-4, 0.0)))
        dr.tau_old[1].copy_(dr.tensor(np.where(np.arange(n) % 3 == 0, -2e-4, 0.0)))
    bc = [fem.DirichletBoundaryCondition(mesh.boundary_nodes, x[mesh.boundary_nodes - 1].copy()) for x in f]
    return dr, bc


# an iteration's increments carry a few FP32 roundings (6e-8) of sums over 27 points and 8 elements
@pytest.mark.parametrize("nel,shear,load", [((1, 1, 1), False, "rest"), ((5, 3, 2), False, "yield"), ((11, 3, 1), False, "yield"),
                                            ((4, 4, 4), True, "yield"), ((33, 2, 1), True, "rest"), ((7, 5, 3), False, "apex"),
                                            ((7, 5, 3), True, "apex")])
def test_increments_match_fp64(nel, shear, load):
    out = []
    for precision in ("fp64", "mixed"):
        dr, bc = state(nel, 3, shear, load)
        v0, P0 = [x.clone() for x in dr.v], dr.P.clone()
        st = fem.solve(dr, bc, dt=0.1, tolerance=1e-9, check_interval=1000, max_iterations=6, throw_on_failure=False,
                       precision=precision)
        out.append(([a - b for a, b in zip(dr.v, v0)] + [dr.P - P0], st["iter"]))
    (ref, it0), (got, it1) = out
    assert it0 == it1
    scale = max(float(x.norm()) for x in ref[:3])
    for a, b in zip(got[:3], ref[:3]):
        assert float((a - b).norm()) <= 5e-6 * scale
    assert float((got[3] - ref[3]).norm()) <= 5e-6 * float(ref[3].norm())
