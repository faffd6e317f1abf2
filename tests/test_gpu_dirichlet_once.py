"""The solves pin the constrained entries once, after the first update: from a start whose
velocities differ from the prescribed ones the device takes the oracle's path."""
import numpy as np
import pytest

import oracle_host as oh
from cases import inclusion_2d_case, vep_layers_case
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,check", [(3, 50), (2, 50), (3, 1)])
def test_start_off_the_prescribed_velocities(dim, check):
    case = vep_layers_case(n=2, seed=0) if dim == 3 else inclusion_2d_case(n=4)
    rng = np.random.default_rng(5)
    case.v = [x + 0.1 * rng.standard_normal(x.shape) for x in case.v]
    dr, hs = case.device_state(fem), case.host_state(oh)
    kw = dict(dt=case.dt, tolerance=1e-9, check_interval=check, max_iterations=60, throw_on_failure=False)
    st = fem.solve(dr, case.bc_device(), **kw)
    ref = hs.solve(**kw)
    assert (st["iter"], st["itPH"]) == (ref["iter"], ref["itPH"])
    # 60 iterations of a contraction in FP64: the summation order moves the fields by ~1e-13
    for c in range(dim):
        scale = np.abs(hs.v[c]).max()
        assert np.abs(dr.v[c].cpu().numpy() - hs.v[c]).max() <= 1e-10 * scale
        dofs, vals = case.bc[c]
        assert np.array_equal(dr.v[c].cpu().numpy()[dofs - 1], vals)
