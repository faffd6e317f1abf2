"""Iterations of the heat-diffusion solve on affine cells, which run on tiles of 32 elements, against
the allocation-free solve, which keeps the per-point geometry and the general kernel."""
import ctypes as C

import numpy as np
import pytest

from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
abi = fem._abi

KW = dict(k=(1.0, 2.5), Cp=(1.0, 1.3), rho0=(1.0, 1.2), alpha=(0.05, 0.02), K=(50.0, 80.0))


# elements: one, a part of a tile, one tile, a tile and one element, several tiles with a part. A
# residual entry sums 8 elements' 27 points × 27 nodes of terms below ~10 times its scale, six
# times over: 1e5 units in the last place
@pytest.mark.parametrize("nel,phases", [((1, 1, 1), "one"), ((5, 3, 1), "mixed"), ((4, 4, 2), "one"), ((11, 3, 1), "mixed"),
                                        ((9, 7, 5), "layers"), ((9, 7, 5), None)])
@pytest.mark.parametrize("sheared,point_source,pressure", [(False, True, True), (True, False, False)])
def test_tiles(nel, phases, sheared, point_source, pressure):
    rng = np.random.default_rng(sum(nel))
    mesh = fem.structured_mixed_mesh(3, nel)
    if sheared:
        c = mesh.coords
        c[:, 0] += 0.2 * c[:, 1]
        c[:, 1] += 0.1 * c[:, 2]
        mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    ph = None if phases is None else {"one": np.full(mesh.nnodes, 2), "mixed": rng.integers(1, 3, mesh.nnodes),
                                      "layers": np.where(mesh.coords[:, 2] < 0.4, 1, 2)}[phases].astype(np.int32)
    fields = {n: torch.as_tensor(rng.uniform(0, 1, mesh.nnodes)) for n in ("T", "source", "P")}
    ip = torch.as_tensor(rng.uniform(0, 1, mesh.nq * mesh.nels), device="cuda")
    bc = fem.DirichletBoundaryCondition(mesh.boundary_nodes[:3], np.array([0.2, 0.4, 0.6]))
    out = []
    for alloc in (True, False):
        th = fem.ThermalDiffusionDR(mesh, phases=ph, eps=1e-30, **KW)
        th.T.copy_(fields["T"]); th.T0.copy_(0.5 * fields["T"]); th.source.copy_(fields["source"])
        if pressure:
            th.P.copy_(fields["P"])
        th.source_ip = ip if point_source else None
        th.set_bc(bc)
        c = abi.ThermalControlsC()
        c.dt, c.Tref, c.tolerance = 0.1, 0.3, 1e-30
        c.max_iterations, c.check_interval, c.throw_on_failure = 6, 4, 0
        lib, h = fem.solver._Handle.get()
        st = abi.ThermalStatsC()
        p = th.problem()
        f = lib.femb200_solve_thermal if alloc else lib.femb200_solve_thermal_noalloc
        assert f(h, C.byref(p), C.byref(c), C.byref(st)) == abi.OK
        assert st.iterations == 6
        out.append((th.T.clone(), th.R.clone()))
    for got, want in zip(*out):
        assert float((got - want).abs().max()) <= 1e-10 * float(want.abs().max())
