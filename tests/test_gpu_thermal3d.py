"""The sum-factorised Hex27 heat-diffusion kernel at the edges of its three-element groups,
with point sources, on distorted cells, against the oracle."""
import numpy as np
import pytest

import oracle_host as oh
from conftest import fem

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

KW = dict(k=(1.0, 2.5), Cp=(1.0, 1.3), rho0=(1.0, 1.2), alpha=(0.05, 0.02), K=(50.0, 80.0))


def distorted(nel, rng):
    mesh = fem.structured_mixed_mesh(3, nel)
    c = mesh.coords
    inner = np.all((c > 1e-12) & (c < 1 - 1e-12), axis=1)
    c[inner] += rng.uniform(-0.07, 0.07, size=(inner.sum(), 3)) / np.array(nel)
    mesh.geo_v, mesh.geo_P = fem.mesh.precompute_geometry(c, mesh.el2n, fem.element_tables(3))
    return mesh


# an entry sums 27 points × 27 nodes of terms below ~10 times its scale: 1e4 units in the last place
@pytest.mark.parametrize("dtype,rtol", [("f64", 1e-11), ("f32", 1e-3)])
@pytest.mark.parametrize("nel,phases", [((1, 1, 1), "one"), ((2, 1, 1), "mixed"), ((5, 2, 1), "mixed"), ((13, 1, 1), "one"),
                                        ((5, 3, 3), "layers")])
def test_thermal_assembly_edges(nel, phases, dtype, rtol):
    rng = np.random.default_rng(sum(nel))
    mesh = distorted(nel, rng)
    ph = {"one": np.full(mesh.nnodes, 2), "mixed": rng.integers(1, 3, mesh.nnodes),
          "layers": np.where(mesh.coords[:, 2] < 0.4, 1, 2)}[phases].astype(np.int32)
    td = torch.float64 if dtype == "f64" else torch.float32
    th, ht = fem.ThermalDiffusionDR(mesh, phases=ph, dtype=td, **KW), oh.HostThermal(mesh, phases=ph, **KW)
    for name in ("T", "T0", "source", "P"):
        x = rng.uniform(0, 1, mesh.nnodes)
        getattr(th, name).copy_(torch.as_tensor(x))
        getattr(ht, name)[:] = x
    ip = rng.uniform(0, 1, mesh.nq * mesh.nels)
    th.source_ip, ht.source_ip = torch.as_tensor(ip, dtype=td, device="cuda"), ip
    for jac in (False, True):
        fem.assemble_thermal_residual(th, 0.1, 0.3, compute_jacobian=jac)
        ht.residual(0.1, 0.3, jac=jac)
        for got, ref in [(th.R, ht.R)] + ([(th.dRdT, ht.dRdT), (th.PC, ht.PC)] if jac else []):
            assert np.abs(got.double().cpu().numpy() - ref).max() <= rtol * np.abs(ref).max()
