"""Heat-diffusion and coupled calls without an array that they need are refused before any kernel runs."""
import ctypes as C

import numpy as np
import pytest

from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi


def thermal(mesh):
    th = fem.ThermalDiffusionDR(mesh)
    th.set_bc(fem.DirichletBoundaryCondition(mesh.boundary_nodes[:3], np.zeros(3)))
    return th


@pytest.mark.parametrize("name", ["T", "T0"])
def test_coupled_needs_the_stokes_temperatures(name):
    case = random_state_case(dim=2, n=2, seed=1, phases="cell")
    dr, th = case.device_state(fem), thermal(case.mesh)
    setattr(dr, name, None)
    with pytest.raises(abi.FemB200Error, match="coupled solve needs T, T0"):
        fem.solve_coupled(th, dr, fem.DirichletBoundaryCondition(case.mesh.boundary_nodes[:3], np.zeros(3)), case.bc_device(),
                          case.dt, max_iterations=1, throw_on_failure=False)


@pytest.mark.parametrize("name", ["el2n", "geo", "T", "T0", "R", "dRdT", "PC", "rate", "R0", "bc_dofs", "bc_vals"])
def test_thermal_needs_its_arrays(name):
    mesh = fem.structured_mixed_mesh(3, (2, 1, 1))
    p = thermal(mesh).problem()
    setattr(p, name, 0)
    lib, h = fem.solver._Handle.get()
    c, st = abi.ThermalControlsC(), abi.ThermalStatsC()
    c.dt, c.tolerance, c.max_iterations, c.check_interval = 0.1, 1e-6, 2, 1
    for f in (lib.femb200_solve_thermal, lib.femb200_solve_thermal_noalloc):
        assert f(h, C.byref(p), C.byref(c), C.byref(st)) == abi.EINVAL
    if name in ("el2n", "geo", "T", "T0", "R", "dRdT", "PC"):
        assert lib.femb200_thermal_residual(h, C.byref(p), 0.1, 0.0, 1) == abi.EINVAL


def test_thermal_needs_a_check_interval():
    mesh = fem.structured_mixed_mesh(3, (2, 1, 1))
    p = thermal(mesh).problem()
    lib, h = fem.solver._Handle.get()
    c, st = abi.ThermalControlsC(), abi.ThermalStatsC()
    c.dt, c.tolerance, c.max_iterations = 0.1, 1e-6, 2
    assert lib.femb200_solve_thermal(h, C.byref(p), C.byref(c), C.byref(st)) == abi.EINVAL
