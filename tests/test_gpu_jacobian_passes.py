"""Kernels that one FP64 assembly of the Jacobian diagnostics launches: on a mesh that is no box the
look for off-diagonal entries and the assembly, no pass that compresses a geometry it cannot use."""
import ctypes as C

import pytest

from cases import random_state_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi


@pytest.mark.parametrize("cells", ["sheared", "distorted"])
def test_launches(cells):
    case = random_state_case(dim=3, n=4, seed=5, phases="cell", plastic=True, distort=cells == "distorted")
    dr = case.device_state(fem)
    fem.assemble_augmented_momentum_jacobian(dr, case.dt)
    lib, h = fem.solver._Handle.get()
    ms, n = (C.c_double * abi.PROF_COUNT)(), (C.c_int64 * abi.PROF_COUNT)()
    assert lib.femb200_profile(h, 1) == abi.OK
    fem.assemble_augmented_momentum_jacobian(dr, case.dt)
    assert lib.femb200_profile_read(h, ms, n) == abi.OK
    lib.femb200_profile(h, 0)
    assert n[abi.PROF_ALL] == 2
