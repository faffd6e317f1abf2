"""Performance cases of the solvers: what a program that uses this framework has it do.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` builds what
the program holds before the call (mesh, state, boundary conditions), `run` makes one pass
through the public entry points, `work` counts what the path cannot do without, and `exact`
computes the same outputs in plain torch in 64 bits.

A solve runs for a fixed number of pseudo-time iterations from a saved initial state, which
`run` copies back first (a time loop that retries a step does the same), so that every pass
does the same work; the tolerances are the ones the solves are used with, which these
iteration counts do not reach. The mixed-precision solves check once, at the end: between
checks the iteration is linear in its step sizes, so that single-precision rounding stays
rounding instead of moving the step sizes that a check derives from it.
"""
from __future__ import annotations

import importlib.util
import math
import os
import sys

import numpy as np
import torch

F64 = torch.float64


def _package():
    """The framework (its directory name is not an identifier: loaded by path)."""
    if "femtools_b200" not in sys.modules:
        d = os.path.join(os.getcwd(), "femtools.jl_b200")
        spec = importlib.util.spec_from_file_location("femtools_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["femtools_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["femtools_b200"]


# ---- the cases ---------------------------------------------------------------------

def listed():
    return [
        # the smallest 3-D solve a user runs (a model being set up): launches and latency
        {"name": "stokes3d_small", "kind": "solve3d", "nx": 6, "ny": 5, "nz": 7, "precision": "fp64", "loaded": False,
         "iterations": 300, "check": 50},
        # the headline workload's mesh and method: layered visco-elasto-plastic 64³, first step
        {"name": "stokes3d_mixed_64", "kind": "solve3d", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed",
         "loaded": False, "iterations": 300, "check": 300},
        # a later step of the 32³ time loop: stored stress near yield, plastic return active
        {"name": "stokes3d_mixed_32_yield", "kind": "solve3d", "nx": 32, "ny": 32, "nz": 32, "precision": "mixed",
         "loaded": True, "iterations": 300, "check": 300},
        # one fused residual assembly on a deformed mesh with nodal phases and temperature
        {"name": "residual_distorted", "kind": "residual", "nx": 40, "ny": 33, "nz": 29, "float32": False},
        # one assembly of the augmented Jacobian diagnostics in the FP64 solve, odd box
        {"name": "jacobian_f64", "kind": "jacobian", "nx": 32, "ny": 31, "nz": 33, "float32": False},
        # 2-D viscous inclusion on 64² (the plain small workload)
        {"name": "stokes2d_inclusion_64", "kind": "solve2d", "problem": "inclusion", "nx": 64, "ny": 64,
         "iterations": 1000, "check": 100},
        # 2-D visco-elasto-plastic shear band on 256², a step of its time loop
        {"name": "stokes2d_shear_band_256", "kind": "solve2d", "problem": "shear_band", "nx": 256, "ny": 256,
         "iterations": 600, "check": 100},
        # the adjoint solve and the viscosity gradient at 32³
        {"name": "adjoint_32", "kind": "adjoint", "nx": 32, "ny": 32, "nz": 32, "iterations": 300},
        # thermal and Stokes iterations together with shear heating at 32³
        {"name": "coupled_32", "kind": "coupled", "nx": 32, "ny": 32, "nz": 32, "iterations": 200, "check": 50},
        # heat diffusion alone, ragged box, two phases
        {"name": "thermal_ragged", "kind": "thermal", "nx": 27, "ny": 35, "nz": 22, "iterations": 200},
        # sinking block of the cell-pressure solver at 32³
        {"name": "cell_pressure_32", "kind": "cell_pressure", "nx": 32, "ny": 32, "nz": 32, "iterations": 1000},
        # one training step of the warm-start network on 8 images of 513² (a 256² mesh's nodes)
        {"name": "network_train_8x513", "kind": "network", "images": 8, "height": 513, "width": 513, "train": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve3d", "solve3d", "residual", "jacobian", "solve2d", "adjoint", "coupled", "thermal",
                       "cell_pressure", "network"])

    def box(lo, hi):
        # three independent sizes round a common one: odd and ragged boxes
        n = _log(rng, lo, hi)
        return {k: max(2, min(hi, int(round(n * rng.uniform(0.8, 1.25))))) for k in ("nx", "ny", "nz")}

    if kind == "solve3d":
        prec = rng.choice(["mixed", "fp64"])
        b = box(5, 56 if prec == "mixed" else 32)
        it = 50 * rng.randint(2, 6)
        return {"kind": kind, **b, "precision": prec, "loaded": rng.random() < 0.5, "iterations": it,
                "check": it if prec == "mixed" else rng.choice([50, 100])}
    if kind in ("residual", "jacobian"):
        return {"kind": kind, **box(6, 48 if kind == "residual" else 32), "float32": rng.random() < 0.3}
    if kind == "solve2d":
        n = _log(rng, 16, 256)
        return {"kind": kind, "problem": rng.choice(["inclusion", "shear_band"]), "nx": n,
                "ny": max(8, int(n * rng.uniform(0.6, 1.0))), "iterations": 50 * rng.randint(4, 10), "check": 100}
    if kind in ("adjoint", "coupled"):
        c = {"kind": kind, **box(6, 32), "iterations": 50 * rng.randint(2, 4)}
        return {**c, "check": 50} if kind == "coupled" else c
    if kind == "thermal":
        return {"kind": kind, **box(6, 32), "iterations": 50 * rng.randint(2, 4)}
    if kind == "cell_pressure":
        return {"kind": kind, **box(6, 32), "iterations": 100 * rng.randint(3, 10)}
    return {"kind": kind, "images": rng.randint(1, 8), "height": _log(rng, 33, 513), "width": _log(rng, 33, 513),
            "train": rng.random() < 0.5}


# ---- meshes and inputs (plain numpy and torch, from the seed alone) ------------------

_HEX = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1),
        (0, -1, -1), (1, 0, -1), (0, 1, -1), (-1, 0, -1), (0, -1, 1), (1, 0, 1), (0, 1, 1), (-1, 0, 1),
        (-1, -1, 0), (1, -1, 0), (1, 1, 0), (-1, 1, 0), (0, 0, -1), (0, -1, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0),
        (0, 0, 1), (0, 0, 0)]
_QUAD = [(-1, -1), (1, -1), (1, 1), (-1, 1), (0, -1), (1, 0), (0, 1), (-1, 0), (0, 0)]
_PNODES = {3: [26, 22, 23, 25], 2: [8, 5, 6]}


def _sizes(case):
    return (case["nx"], case["ny"], case["nz"]) if "nz" in case else (case["nx"], case["ny"])


class _Box:
    """Structured quadratic mesh of the unit square or cube: nodes x fastest, 0-based connectivity."""

    def __init__(self, nel, move=None):
        self.nel, self.dim = tuple(nel), len(nel)
        loc = np.array(_HEX if self.dim == 3 else _QUAD)
        pts = [2 * n + 1 for n in self.nel]
        axes = [np.arange(p, dtype=np.float64) / (p - 1) for p in pts]
        g = np.meshgrid(*axes[::-1], indexing="ij")
        self.coords = np.stack([x.ravel() for x in g[::-1]], axis=1)
        idx = np.meshgrid(*[np.arange(n) for n in self.nel[::-1]], indexing="ij")
        idx = [i.ravel() for i in idx[::-1]]
        node, stride = 0, 1
        for d in range(self.dim):
            node = node + (2 * idx[d][:, None] + 1 + loc[None, :, d]) * stride
            stride *= pts[d]
        self.el2n = node.astype(np.int32)
        self.boundary = np.nonzero(((self.coords == 0.0) | (self.coords == 1.0)).any(axis=1))[0]
        if move is not None:
            self.coords = move(self.coords)
        ncorner = 8 if self.dim == 3 else 4
        self.centre = self.coords[self.el2n[:, :ncorner]].mean(axis=1)
        self.nels, self.nnodes, self.np = len(self.el2n), len(self.coords), self.dim + 1

    def walls(self, axis, both=True):
        x = self.coords[:, axis]
        return np.nonzero((x == 0.0) | ((x == 1.0) & both))[0]

    def mesh(self):
        """The framework's mesh of this box, geometry by its own assembly."""
        fem = _package()
        el2n = self.el2n + 1
        geo_v, geo_P = fem.precompute_geometry(self.coords, el2n, self.dim)
        dofs = (np.arange(self.nels * self.np, dtype=np.int64).reshape(self.nels, self.np) + 1).astype(np.int32)
        return fem.MixedMesh(self.dim, self.nel, self.coords, el2n, dofs, el2n[:, _PNODES[self.dim]].copy(), geo_v,
                             geo_P, (self.boundary + 1).astype(np.int32))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=F64)


def _rand(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=F64)


def _layered(case, seed):
    """Three horizontal layers, pure-shear walls; `loaded` starts from a stored stress that
    brings part of the points to yield, as the later steps of a time loop do."""
    rng = np.random.default_rng(seed)
    box = _Box(_sizes(case))
    z1, z2 = np.sort(rng.uniform(0.3, 0.7, size=2))
    eta, C = 10.0 ** rng.uniform(0.0, 3.0, size=3), rng.uniform(0.3, 1.0, size=3)
    zc = box.centre[:, 2]
    phase = np.where(zc < z1, 0, np.where(zc < z2, 1, 2))
    inf = [math.inf] * 3
    mat = dict(eta=list(eta), eta_b=[10.0] * 3, G=[1.0] * 3, alpha=[0.0] * 3, rho0=[1.0] * 3, K=[10.0] * 3,
               g=[0.0, 0.0, -1.0], Tref=0.0, inf=inf)
    pl = dict(phi=[math.radians(30)] * 3, psi=[0.0] * 3, C=list(C), eta_reg=[0.1 if case["loaded"] else 1e-2] * 3, Kb=[10.0] * 3)
    x, y, z = box.coords.T
    v = [x - 0.5, np.zeros_like(y), -(z - 0.5)]
    bc = [(box.boundary, f[box.boundary].copy()) for f in v]
    nqe = 27 * box.nels
    told = [torch.zeros(nqe, device="cuda", dtype=F64) for _ in range(6)]
    if case["loaded"]:
        g = _gen(seed)
        amp = torch.as_tensor(0.8 * math.cos(math.radians(30)) * C[phase], device="cuda").repeat_interleave(27)
        told[0] = amp * (1 + 0.05 * _randn(g, nqe))
        told[2] = -told[0]
        for c in (3, 4, 5):
            told[c] = 0.03 * amp * _randn(g, nqe)
    return dict(box=box, mat=mat, plastic=pl, phase=phase, v=v, bc=bc, told=told, dt=0.1)


def _plane(case, seed):
    """The 2-D workloads: a viscous inclusion under gravity, or a shear band round a weak seed."""
    rng = np.random.default_rng(seed)
    box = _Box(_sizes(case))
    cx, cy = box.centre.T
    x, y = box.coords.T
    nqe = 9 * box.nels
    if case["problem"] == "inclusion":
        ox, oy, r = rng.uniform(0.45, 0.55), rng.uniform(0.45, 0.55), rng.uniform(0.09, 0.12)
        phase = (np.hypot(cx - ox, cy - oy) < r).astype(np.int64)
        mat = dict(eta=[1.0, 10.0 ** rng.uniform(2.5, 3.0)], eta_b=[math.inf] * 2, G=[math.inf] * 2, alpha=[0.0] * 2,
                   rho0=[1.0, 1.1], K=[math.inf] * 2, g=[0.0, -1.0], Tref=0.0)
        bc = [(box.walls(d), np.zeros(len(box.walls(d)))) for d in range(2)]
        return dict(box=box, mat=mat, plastic=None, phase=phase, v=[np.zeros(box.nnodes)] * 2, bc=bc,
                    told=[torch.zeros(nqe, device="cuda", dtype=F64) for _ in range(3)], dt=1.0)
    ox, oy = rng.uniform(0.4, 0.6, size=2)
    phase = (np.hypot(cx - ox, cy - oy) < 0.02 + 0.5 / min(box.nel)).astype(np.int64)
    mat = dict(eta=[1e2, 1.0], eta_b=[10.0] * 2, G=[1.0] * 2, alpha=[0.0] * 2, rho0=[1.0] * 2, K=[10.0] * 2,
               g=[0.0, 0.0], Tref=0.0)
    pl = dict(phi=[math.radians(30)] * 2, psi=[0.0] * 2, C=[0.5] * 2, eta_reg=[1.0] * 2, Kb=[10.0] * 2)
    v = [y - 0.5, np.zeros_like(y)]
    bc = [(box.boundary, f[box.boundary].copy()) for f in v]
    g = _gen(seed)
    told = [0.02 * _randn(g, nqe), torch.zeros(nqe, device="cuda", dtype=F64), 0.4 * (1 + 0.03 * _randn(g, nqe))]
    return dict(box=box, mat=mat, plastic=pl, phase=phase, v=v, bc=bc, told=told, dt=0.1)


def _element_state(case, seed):
    """One assembly: a random state about yield, three phases; the residual on a deformed mesh
    with nodal phases, the Jacobian on the box the solves use, one phase per cell."""
    rng = np.random.default_rng(seed)
    deformed = case["kind"] == "residual"
    nel = _sizes(case)

    def move(c):
        out = c.copy()
        inner = ((c > 0.0) & (c < 1.0)).all(axis=1)
        h = 1.0 / (2 * np.array(nel))
        out[inner] += rng.uniform(-0.15, 0.15, size=(inner.sum(), 3)) * h
        return out

    box = _Box(nel, move if deformed else None)
    # contrasts below 2.5: the quadratic interpolation of nodal phases undershoots, and stays positive
    mat = dict(eta=list(10 ** rng.uniform(0, 0.4, 3)), eta_b=list(rng.uniform(15, 35, 3)), G=list(rng.uniform(1, 2.5, 3)),
               alpha=list(rng.uniform(0.04, 0.1, 3)), rho0=list(rng.uniform(1, 2, 3)), K=list(rng.uniform(40, 100, 3)),
               g=[0.0, 0.3, -1.0], Tref=0.1)
    pl = dict(phi=list(rng.uniform(0.3, 0.6, 3)), psi=list(rng.uniform(0.1, 0.2, 3)), C=list(rng.uniform(0.12, 0.3, 3)),
              eta_reg=list(rng.uniform(0.04, 0.1, 3)), Kb=list(rng.uniform(4, 10, 3)))
    g, nn, nP, nqe = _gen(seed), box.nnodes, 4 * box.nels, 27 * box.nels
    x = torch.as_tensor(box.coords, device="cuda")
    f32 = case["float32"]
    r32 = (lambda t: t.float().double()) if f32 else (lambda t: t)     # inputs a 32-bit state holds exactly
    v = [r32(x[:, c] * s + 0.05 * torch.sin(7 * x[:, (c + 1) % 3]) + 0.2 / max(nel) * _randn(g, nn))
         for c, s in zip(range(3), (1.0, 0.2, -1.0))]
    out = dict(box=box, mat=mat, plastic=pl, v=v, bc=None, dt=0.7, P=r32(0.3 * _randn(g, nP)), P0=r32(0.3 * _randn(g, nP)),
               T=r32(_randn(g, nP)), T0=r32(_randn(g, nP)), told=[r32(0.1 * _randn(g, nqe)) for _ in range(6)],
               gammaP=r32(_rand(g, 1.0, 5.0, nP)), M_P=r32(_rand(g, 0.01, 0.1, nP)))
    if deformed:
        out["phase_nodes"] = rng.integers(0, 3, nn)
        out["phase_dofs"] = rng.integers(0, 3, nP)
    else:
        out["phase"] = rng.integers(0, 3, box.nels)
    return out


def _hot(case, seed):
    """Hot viscous convection set-up: T falls from 1 (bottom) to 0 (top) with noise, a random
    log-viscosity per element, free slip on sides and bottom, free top."""
    rng = np.random.default_rng(seed)
    box = _Box(_sizes(case))
    h = 1.0 / box.nel[2]
    Tc = 1.0 - box.centre[:, 2]
    Td = np.stack([Tc, Tc, Tc, Tc - 0.5 * h], axis=1) + rng.normal(0.0, 0.01, size=(box.nels, 4))
    delta = rng.normal(0.0, 0.1, size=box.nels)
    tab = _Tables(3)
    T = torch.as_tensor(Td, device="cuda")
    eta_ip = (torch.exp(-0.1 * (T @ tab.NP.T)) * torch.exp(torch.as_tensor(delta, device="cuda"))[:, None]).reshape(-1)
    mat = dict(eta=[1.0], eta_b=[10.0], G=[math.inf], alpha=[0.1], rho0=[1.0], K=[math.inf], g=[0.0, 0.0, -1.0],
               Tref=0.0)
    bc = []
    for d in range(3):
        w = box.walls(d, both=d < 2)
        bc.append((w, np.zeros(len(w))))
    z = box.coords[:, 2]
    top = np.nonzero(z == 1.0)[0]
    out = dict(box=box, mat=mat, plastic=None, phase=np.zeros(box.nels, dtype=np.int64), bc=bc, dt=1.0, T=T.reshape(-1),
               T0=T.reshape(-1).clone(), eta_ip=eta_ip, told=[torch.zeros(27 * box.nels, device="cuda", dtype=F64)] * 6,
               top=top, v=[np.zeros(box.nnodes)] * 3)
    g = _gen(seed)
    if case["kind"] == "adjoint":
        obj = torch.zeros(3, box.nnodes, device="cuda", dtype=F64)
        obj[:, torch.as_tensor(top, device="cuda")] = 0.02 * _randn(g, 3, len(top))
        out["objective"] = [o.contiguous() for o in obj]
        x = torch.as_tensor(box.coords, device="cuda")
        out["v"] = [0.01 * torch.sin(3 * x[:, (c + 1) % 3]) for c in range(3)]
        out["P"] = 0.1 * _randn(g, 4 * box.nels)
    return out


def _heat(case, seed):
    """Heat diffusion: two phases by node, a warm blob, fixed top and bottom temperatures."""
    rng = np.random.default_rng(seed)
    box = _Box(_sizes(case))
    x, y, z = box.coords.T
    phase = (z > rng.uniform(0.3, 0.7)).astype(np.int64)
    c = rng.uniform(0.3, 0.7, size=3)
    T = 1.0 - z + np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / 0.02) + rng.normal(0, 0.01, box.nnodes)
    bottom, top = np.nonzero(z == 0.0)[0], np.nonzero(z == 1.0)[0]
    nodes = np.concatenate([bottom, top])
    vals = np.concatenate([np.ones(len(bottom)), np.zeros(len(top))])
    mat = dict(k=[1.0, rng.uniform(1.5, 4.0)], Cp=[1.0, rng.uniform(0.8, 1.2)], rho0=[1.0, rng.uniform(1.0, 1.3)],
               alpha=[0.03, 0.01], K=[100.0, 50.0])
    return dict(box=box, phase_nodes=phase, T=T, source=rng.uniform(0.0, 1.0, box.nnodes),
                P=rng.uniform(0.0, 1.0, box.nnodes), bc=(nodes, vals), mat=mat, dt=0.05, Tref=0.0)


def _block(case, seed):
    """A dense viscous block sinking in a matrix, free slip on every wall."""
    rng = np.random.default_rng(seed)
    box = _Box(_sizes(case))
    o, w = rng.uniform(0.45, 0.55, size=3), rng.uniform(0.2, 0.28)
    phase = (np.abs(box.centre - o) < w).all(axis=1).astype(np.int64)
    mat = dict(eta=[1.0, 10.0 ** rng.uniform(1.5, 2.0)], rho0=[1.0, rng.uniform(1.3, 1.5)], g=[0.0, 0.0, -1.0])
    bc = [(box.walls(d), np.zeros(len(box.walls(d)))) for d in range(3)]
    return dict(box=box, phase=phase, mat=mat, bc=bc)


_INPUTS = {"solve3d": _layered, "solve2d": _plane, "residual": _element_state, "jacobian": _element_state,
           "adjoint": _hot, "coupled": _hot, "thermal": _heat, "cell_pressure": _block}


# ---- the framework's side ----------------------------------------------------------------

def _stokes(inp, dtype=None):
    fem = _package()
    m, p, box = inp["mat"], inp["plastic"], inp["box"]
    mat = fem.StokesMaterial(eta=m["eta"], eta_b=m["eta_b"], G=m["G"], alpha=m["alpha"], rho0=m["rho0"], K=m["K"],
                             g=m["g"], Tref=m["Tref"])
    pl = fem.DruckerPrager.from_angles(p["phi"], p["psi"], p["C"], p["eta_reg"], p["Kb"]) if p else None
    abi = fem._abi
    if "phase" in inp:
        ph = (inp["phase"] + 1).astype(np.int32)
        kw = dict(phases_v=ph, phases_v_layout=abi.PHASE_CELL, phases_P=ph, phases_P_layout=abi.PHASE_CELL)
    else:
        kw = dict(phases_v=inp["phase_nodes"] + 1, phases_P=inp["phase_dofs"] + 1)
    dr = fem.StokesDR(box.mesh(), mat, pl, dtype=dtype, **kw)
    for c in range(box.dim):
        dr.v[c].copy_(torch.as_tensor(inp["v"][c], device="cuda"))
    for name in ("P", "P0", "T", "T0", "gammaP", "M_P"):
        if name in inp:
            getattr(dr, name).copy_(inp[name])
    for c, t in enumerate(inp["told"]):
        dr.tau_old[c].copy_(t)
    if "eta_ip" in inp:
        dr.viscosity_ip = inp["eta_ip"].to(dr.dtype).contiguous()
    bc = None
    if inp["bc"] is not None:
        bc = [fem.DirichletBoundaryCondition((n + 1).astype(np.int32), x) for n, x in inp["bc"]]
    return dr, bc


def prepare(case, seed):
    fem = _package()
    kind = case["kind"]
    if kind == "network":
        H, W, B = case["height"], case["width"], case["images"]
        net = fem.warmstart.WarmStartNet(seed=int(seed))
        x, target = _images(case, seed)
        return dict(case=case, net=net, x=x, target=target)
    inp = _INPUTS[kind](case, seed)
    if kind == "thermal":
        m = inp["mat"]
        th = fem.ThermalDiffusionDR(inp["box"].mesh(), k=m["k"], Cp=m["Cp"], rho0=m["rho0"], alpha=m["alpha"], K=m["K"],
                                    phases=inp["phase_nodes"] + 1)
        for name in ("T", "source", "P"):
            getattr(th, name).copy_(torch.as_tensor(inp[name], device="cuda"))
        th.T0.copy_(th.T)
        n, x = inp["bc"]
        return dict(case=case, th=th, bc=fem.DirichletBoundaryCondition((n + 1).astype(np.int32), x), inp=inp)
    if kind == "cell_pressure":
        m = inp["mat"]
        mesh = inp["box"].mesh()
        mesh.geo_v = mesh.geo_v.cpu().numpy()
        dr = fem.CellPressureStokesDR(mesh, fem.StokesMaterial(eta=m["eta"], rho0=m["rho0"], g=m["g"]),
                                      inp["phase"] + 1)
        bc = [fem.DirichletBoundaryCondition((n + 1).astype(np.int32), x) for n, x in inp["bc"]]
        return dict(case=case, dr=dr, bc=bc)
    dr, bc = _stokes(inp, torch.float32 if case.get("float32") else F64)
    s = dict(case=case, dr=dr, bc=bc, dt=inp["dt"], v0=[x.clone() for x in dr.v], P0=dr.P.clone())
    if kind == "adjoint":
        s["objective"] = inp["objective"]
        fem.assemble_viscosity_weighted_pressure_scaling(dr, 50.0, inp["dt"])
    if kind == "coupled":
        box = inp["box"]
        th = fem.ThermalDiffusionDR(dr.mesh, k=(1.0,), Cp=(1.0,), rho0=(1.0,), alpha=(0.1,), K=(math.inf,))
        s["T0"] = torch.as_tensor(_nodal_T(box, seed), device="cuda")
        th.T0.copy_(s["T0"])
        n, x = _thermal_walls(box)
        s.update(th=th, bc_T=fem.DirichletBoundaryCondition((n + 1).astype(np.int32), x))
    torch.cuda.synchronize()
    return s


def _nodal_T(box, seed):
    return 1.0 - box.coords[:, 2] + np.random.default_rng(seed + 1).normal(0.0, 0.01, box.nnodes)


def _thermal_walls(box):
    z = box.coords[:, 2]
    lo, hi = np.nonzero(z == 0.0)[0], np.nonzero(z == 1.0)[0]
    return np.concatenate([lo, hi]), np.concatenate([np.ones(len(lo)), np.zeros(len(hi))])


def run(s):
    fem = _package()
    case = s["case"]
    kind = case["kind"]
    if kind in ("solve3d", "solve2d"):
        dr = s["dr"]
        for c in range(dr.mesh.dim):
            dr.v[c].copy_(s["v0"][c])
        dr.P.copy_(s["P0"])
        st = fem.solve(dr, s["bc"], dt=s["dt"], tolerance=1e-8, check_interval=case["check"],
                       max_iterations=case["iterations"], iter_max=2_000_000, throw_on_failure=False,
                       precision=case.get("precision", "fp64"))
        return {"v": dr.v, "P": dr.P, "iterations": st["iter"]}
    if kind == "residual":
        fem.assemble_stokes_residuals(s["dr"], s["dt"])
        return {"Rv": s["dr"].Rv, "RP": s["dr"].RP, "Pnum": s["dr"].Pnum}
    if kind == "jacobian":
        fem.assemble_augmented_momentum_jacobian(s["dr"], s["dt"])
        return {"rows": s["dr"].dRdv, "diag": s["dr"].PC}
    if kind == "adjoint":
        dr = s["dr"]
        lv, lP, st = fem.solve_adjoint(dr, s["bc"], s["dt"], s["objective"], max_iterations=case["iterations"],
                                       check_interval=50, throw_on_failure=False)
        g = fem.viscosity_sensitivity(dr, s["dt"], lv, lP)
        return {"lam_v": lv, "lam_P": lP, "sensitivity": g, "iterations": st["iter"]}
    if kind == "coupled":
        dr, th = s["dr"], s["th"]
        for c in range(3):
            dr.v[c].copy_(s["v0"][c])
        dr.P.copy_(s["P0"])
        th.T.copy_(s["T0"])
        st, phi = fem.solve_coupled(th, dr, s["bc_T"], s["bc"], s["dt"], Tref=0.0, shear_heating=True, tolerance=1e-8,
                                    max_iterations=case["iterations"], check_interval=case["check"],
                                    throw_on_failure=False)
        return {"v": dr.v, "P": dr.P, "T": th.T, "iterations": st["iter"]}
    if kind == "thermal":
        th, inp = s["th"], s["inp"]
        th.T.copy_(th.T0)
        th.rate.zero_()
        st = fem.solve_thermal(th, s["bc"], inp["dt"], Tref=inp["Tref"], tolerance=1e-12,
                               max_iterations=case["iterations"], check_interval=50, throw_on_failure=False)
        return {"T": th.T, "R": th.R, "iterations": st["iterations"]}
    if kind == "cell_pressure":
        dr = s["dr"]
        for c in range(3):
            dr.v[c].zero_()
        dr.P.zero_()
        st = fem.cellpressure.solve_cell_pressure(dr, s["bc"], tolerance=1e-8, max_iterations=case["iterations"],
                                                  check_interval=100, throw_on_failure=False)
        return {"v": dr.v, "P": dr.P, "iterations": st["iterations"]}
    net, B, H, W = s["net"], case["images"], case["height"], case["width"]
    if not case["train"]:
        out, _ = net.forward(s["x"], B, H, W)
        return {"out": out}
    net.zero_grad()
    out, acts = net.forward(s["x"], B, H, W, keep=True)
    loss, dy = net.loss_grad(out, s["target"], B * H * W, 1.0 / (B * H * W))
    net.backward(acts, dy, B, H, W)
    net.adam()
    return {"loss": loss, "gw": [L["gw"] for L in net.layers], "gb": [L["gb"] for L in net.layers]}


# ---- what the path cannot do without ------------------------------------------------

def work(case):
    """An iterative solve needs its state once per iteration (every iteration reads the last
    one's velocities); a single assembly or network pass reads its inputs and writes its
    outputs once. Flops are those of the sum-factorised element sweep."""
    kind = case["kind"]
    if kind == "network":
        px = case["images"] * case["height"] * case["width"]
        w = 9 * (16 * 32 + 4 * 32 * 32 + 32 * 16)
        passes = 3 if case["train"] else 1
        # activations written once and, in training, read once more; the data gradients are new
        acts = px * (16 + 5 * 32) * 2
        return {"bytes": acts * passes + px * 16 * 4, "flops": 2.0 * w * px * passes}
    nel = _sizes(case)
    ne = math.prod(nel)
    nn = math.prod(2 * n + 1 for n in nel)
    it = case.get("iterations", 1)
    if kind in ("residual", "jacobian"):
        w = 4 if case["float32"] else 8
        per = nn * 3 * w * (2 if kind == "residual" else 3) + ne * 4 * w * 8 + ne * 27 * 4 + ne * 27 * 6 * w
        per += ne * 27 * 11 * w
        return {"bytes": per, "flops": ne * (12e3 if kind == "residual" else 81 * 6e3)}
    if kind == "solve2d":
        per = nn * 2 * 8 * 5 + ne * (3 * 8 * 6 + 9 * 4 + 27 * 8)
        return {"bytes": per * it, "flops": ne * 2.5e3 * it}
    if kind == "thermal":
        return {"bytes": (nn * 8 * 7 + ne * 27 * 4) * it, "flops": ne * 6e3 * it}
    if kind == "cell_pressure":
        return {"bytes": (nn * 3 * 8 * 4 + ne * (4 * 8 * 4 + 27 * 4)) * it, "flops": ne * 9e3 * it}
    if kind == "adjoint":
        return {"bytes": (nn * 3 * 8 * 6 + ne * (4 * 8 * 4 + 27 * 4 + 27 * 8)) * it, "flops": ne * 13e3 * it}
    mixed = case.get("precision") == "mixed"
    w = 4 if mixed else 8
    per = nn * 3 * w * 5 + ne * (4 * w * 6 + 27 * 4) + ne * 27 * (w if mixed else 6 * w)
    flops = ne * 12e3
    if kind == "coupled":
        per += nn * 8 * 7 + ne * 27 * 8
        flops += ne * 6e3
    return {"bytes": per * it, "flops": flops * it}


# ---- the same in plain torch, 64 bits -----------------------------------------------

class _Tables:
    """Quadratic tensor basis at the 3-point Gauss rule and the linear pressure basis."""

    def __init__(self, dim):
        loc = np.array(_HEX if dim == 3 else _QUAD)
        a = math.sqrt(3.0 / 5.0)
        p1, w1 = np.array([-a, 0.0, a]), np.array([5.0, 8.0, 5.0]) / 9.0
        q = np.arange(3 ** dim)
        i = np.stack([(q // 3 ** d) % 3 for d in range(dim)], axis=1)
        x = p1[i]
        n = loc[None, :, :]
        X = x[:, None, :]
        L = np.where(n == 0, 1 - X * X, X * (X + n) * 0.5)
        D = np.where(n == 0, -2 * X, X + 0.5 * n)
        dN = np.stack([np.prod(np.concatenate([L[..., :d], D[..., d:d + 1], L[..., d + 1:]], axis=-1), axis=-1)
                       for d in range(dim)], axis=-1)
        t = lambda z: torch.as_tensor(np.ascontiguousarray(z), device="cuda", dtype=F64)
        self.N, self.dN, self.w = t(np.prod(L, axis=-1)), t(dN), t(np.prod(w1[i], axis=1))
        self.NP = t(np.concatenate([1 - x.sum(axis=1, keepdims=True), x], axis=1))
        self.x = t(x)
        self.dim, self.nq, self.nv = dim, len(q), len(loc)


class _Mesh:
    """Gradients and their transpose on a box's elements: fields are (…, elements, points)."""

    def __init__(self, box):
        self.t = _Tables(box.dim)
        self.dim, self.ne, self.nn = box.dim, box.nels, box.nnodes
        self.el = torch.as_tensor(box.el2n.astype(np.int64), device="cuda")
        X = torch.as_tensor(box.coords, device="cuda")
        d = self.dim
        xe = X[self.el]                                                       # e a i
        J = torch.einsum("eai,qaj->eqij", xe, self.t.dN)
        self.Ji = [[None] * d for _ in range(d)]
        inv = _inverse(J)
        det = _det(J)
        for r in range(d):
            for c in range(d):
                self.Ji[r][c] = inv[r][c].contiguous()                        # ∂ξ_r/∂x_c
        self.dO = det.abs() * self.t.w
        self.G = self.t.dN.permute(1, 2, 0).reshape(self.t.nv, d * self.t.nq).contiguous()   # a, (d q)

    def gradient(self, u):
        """[∂u/∂x_k] of a nodal field."""
        gr = (u[self.el] @ self.G).view(self.ne, self.dim, self.t.nq)
        return [sum(gr[:, r] * self.Ji[r][k] for r in range(self.dim)) for k in range(self.dim)]

    def value(self, u):
        return u[self.el] @ self.t.N.T

    def scatter(self, flux, load=None):
        """Σ_q ∇N_a·flux dΩ (+ N_a load dΩ) added over the elements."""
        F = torch.stack([sum(self.Ji[r][k] * flux[k] for k in range(self.dim)) * self.dO for r in range(self.dim)], dim=1)
        R = F.reshape(self.ne, -1) @ self.G.T
        if load is not None:
            R = R + (load * self.dO) @ self.t.N
        return torch.zeros(self.nn, device="cuda", dtype=F64).index_add_(0, self.el.reshape(-1), R.reshape(-1))

    def physical(self, rows):
        """∇N of some elements: (element, point, node, direction)."""
        return torch.stack([sum(self.Ji[r][k][rows][:, :, None] * self.t.dN[None, :, :, r] for r in range(self.dim))
                            for k in range(self.dim)], dim=-1)


def _det(J):
    g = lambda i, j: J[..., i, j]
    if J.shape[-1] == 2:
        return g(0, 0) * g(1, 1) - g(0, 1) * g(1, 0)
    return (g(0, 0) * (g(1, 1) * g(2, 2) - g(1, 2) * g(2, 1)) - g(0, 1) * (g(1, 0) * g(2, 2) - g(1, 2) * g(2, 0))
            + g(0, 2) * (g(1, 0) * g(2, 1) - g(1, 1) * g(2, 0)))


def _inverse(J):
    d, det = J.shape[-1], _det(J)
    g = lambda i, j: J[..., i, j]
    if d == 2:
        return [[g(1, 1) / det, -g(0, 1) / det], [-g(1, 0) / det, g(0, 0) / det]]
    o = lambda i: [k for k in range(3) if k != i]
    sign = lambda i, j: 1.0 if (i + j) % 2 == 0 else -1.0
    return [[sign(r, c) * (g(o(c)[0], o(r)[0]) * g(o(c)[1], o(r)[1]) - g(o(c)[0], o(r)[1]) * g(o(c)[1], o(r)[0])) / det
             for c in range(3)] for r in range(3)]


_EPS2 = np.finfo(np.float64).eps ** 2
_VOIGT = {3: [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)], 2: [(0, 0), (1, 1), (0, 1)]}


class _Stokes:
    """Augmented visco-elasto-plastic Stokes residual, its Jacobian diagnostics and the DR loop."""

    def __init__(self, inp):
        box = inp["box"]
        self.m = m = _Mesh(box)
        self.box, self.dim, self.dt, t = box, box.dim, inp["dt"], m.t
        ne, mat, pl = m.ne, inp["mat"], inp["plastic"]
        dev = lambda x: torch.as_tensor(np.asarray(x, dtype=np.float64), device="cuda")
        if "phase" in inp:
            ph = torch.as_tensor(inp["phase"], device="cuda")
            nodes, dofs = ph[:, None].expand(ne, t.nv), ph[:, None].expand(ne, box.np)
        else:
            nodes = torch.as_tensor(inp["phase_nodes"], device="cuda")[m.el]
            dofs = torch.as_tensor(inp["phase_dofs"], device="cuda").view(ne, box.np)
        at = lambda vals: dev(vals)[nodes] @ t.N.T
        atP = lambda vals: dev(vals)[dofs] @ t.NP.T
        self.eta = inp["eta_ip"].view(ne, t.nq) if "eta_ip" in inp else at(mat["eta"])
        self.eta_pc = (self.eta if "eta_ip" in inp else dev(mat["eta"])[nodes]).amax(dim=1, keepdim=True)
        self.iG = at([1.0 / x for x in mat["G"]])
        self.rho0, self.alpha, self.beta = at(mat["rho0"]), at(mat["alpha"]), at([1.0 / x for x in mat["K"]])
        self.bulk_inf = all(math.isinf(x) for x in mat["eta_b"])
        self.bulk = None if self.bulk_inf else atP(mat["eta_b"])
        self.alphaP = atP(mat["alpha"])
        self.g, self.Tref = mat["g"], mat["Tref"]
        self.pl = None
        if pl:
            self.pl = dict(cC=at(np.cos(pl["phi"])) * at(pl["C"]), s=at(np.sin(pl["phi"])),
                           rest=at(pl["eta_reg"]) + at(pl["Kb"]) * self.dt * at(np.sin(pl["psi"])) * at(np.sin(pl["phi"])))
        self.told = [x.view(ne, t.nq) for x in inp["told"]]
        z = torch.zeros(ne, box.np, device="cuda", dtype=F64)
        f = lambda name: inp[name].view(ne, box.np) if name in inp else z
        self.P0, self.T, self.T0, self.gP, self.MP = f("P0"), f("T"), f("T0"), f("gammaP"), f("M_P")
        self.inv_bulk = at([1.0 / x for x in mat["eta_b"]])

    def scaling(self, factor=50.0):
        t = self.m.t
        num = factor * self.eta
        phys = torch.where(self.inv_bulk == 0, num, self.dt / self.inv_bulk)
        w = self.m.dO[:, :, None] * (t.NP ** 2)[None]
        self.MP = w.sum(dim=1)
        self.gP = (w * (phys * num / (phys + num))[:, :, None]).sum(dim=1) / self.MP

    def stress(self, gr, Peq, eta):
        """τ (Voigt) from the velocity gradient at the points, and the plastic branch."""
        d = self.dim
        etave = 1.0 / (1.0 / eta + self.iG / self.dt)
        tr = sum(gr[c][c] for c in range(d)) / 3.0
        ed = [gr[i][i] - tr if i == j else 0.5 * (gr[i][j] + gr[j][i]) for i, j in _VOIGT[d]]
        tt = [2 * etave * (e + o * self.iG / (2 * self.dt)) for e, o in zip(ed, self.told)]
        if self.pl is None:
            return tt
        n = d
        sq = sum(x * x for x in tt[:n])
        if d == 2:
            sq = sq + (tt[0] + tt[1]) ** 2
        tII = torch.sqrt(0.5 * sq + sum(x * x for x in tt[n:]) + _EPS2)
        F = tII - self.pl["cC"] - self.pl["s"] * Peq
        lam = torch.where(F > 0, F / (etave + self.pl["rest"]), torch.zeros_like(F))
        f = 2 * etave * lam / (tII + _EPS2)
        if d == 2:
            return [tt[0] - f * (2 * tt[0] + tt[1]) / 2, tt[1] - f * (tt[0] + 2 * tt[1]) / 2, tt[2] - f * tt[2]]
        return [x - 0.5 * f * x for x in tt[:3]] + [x - f * x for x in tt[3:]]

    def residual(self, v, P, pnum=True):
        m, t, d, dt = self.m, self.m.t, self.dim, self.dt
        gr = [m.gradient(u) for u in v]
        Pe = P.view(m.ne, -1)
        f = -sum(gr[c][c] for c in range(d))
        if not self.bulk_inf:
            f = f - ((Pe - self.P0) @ t.NP.T) / (self.bulk * dt)
        f = f + self.alphaP * ((self.T - self.T0) @ t.NP.T) / dt
        RP = (f * m.dO) @ t.NP
        Pn = self.gP * RP / self.MP if pnum else torch.zeros_like(RP)
        Pq = Pe @ t.NP.T
        tau = self.stress(gr, Pq, self.eta)
        Pt = Pq + Pn @ t.NP.T
        rho = self.rho0 * (1 - self.alpha * (self.T @ t.NP.T - self.Tref) + self.beta * Pq)
        s = [[None] * d for _ in range(d)]
        for (i, j), x in zip(_VOIGT[d], tau):
            s[i][j] = s[j][i] = x - Pt if i == j else x
        Rv = [m.scatter(s[c], -rho * self.g[c] if self.g[c] else None) for c in range(d)]
        self.last = (gr, tau)
        return Rv, RP.reshape(-1), Pn.reshape(-1)

    def heating(self, v, P):
        gr = [self.m.gradient(u) for u in v]
        tau = self.stress(gr, P.view(self.m.ne, -1) @ self.m.t.NP.T, self.eta)
        out = 0.0
        for (i, j), x, o in zip(_VOIGT[3], tau, self.told):
            k = 1.0 if i == j else 2.0
            out = out + (x * gr[i][i] if i == j else x * (gr[i][j] + gr[j][i]))
            out = out - k * x * (x - o) * self.iG / (2 * self.dt)
        return out

    def jacobian(self, v, P, chunk=4096):
        """Absolute row sums and |diagonal| of the element Jacobians, added over the elements."""
        m, t, d = self.m, self.m.t, self.dim
        gr = [m.gradient(u) for u in v]
        Pq = P.view(m.ne, -1) @ t.NP.T
        rows = torch.zeros(d, m.nn, device="cuda", dtype=F64)
        diag = torch.zeros_like(rows)
        eta = self.eta_pc.expand(m.ne, t.nq)
        tang = []
        for a in range(d):
            for b in range(d):
                e = [[torch.ones_like(Pq) if (i, j) == (a, b) else torch.zeros_like(Pq) for j in range(d)] for i in range(d)]
                tang.append(_directional(lambda g: self.stress(g, Pq, eta), gr, e))
        # tang[(a, b)][voigt]: ∂τ/∂(∂v_a/∂x_b)
        nv = t.nv
        if d == 2:
            chunk = 1 << 16
        for s0 in range(0, m.ne, chunk):
            r = slice(s0, min(s0 + chunk, m.ne))
            n = r.stop - r.start
            dN = m.physical(r)                                               # e q a k
            dO = m.dO[r]
            BP = -torch.einsum("eq,qp,eqak->epak", dO, t.NP, dN)             # ∂RP_p/∂v_(a, k)
            pn = torch.einsum("qp,epak->eqak", t.NP, BP * (self.gP / self.MP)[r][:, :, None, None])
            J = torch.empty(n, nv, d, nv, d, device="cuda", dtype=F64)       # e i c b j
            for j in range(d):
                sig = [[0.0] * d for _ in range(d)]
                for w, (i1, i2) in enumerate(_VOIGT[d]):
                    x = sum(tang[j * d + k][w][r][:, :, None] * dN[:, :, :, k] for k in range(d))
                    sig[i1][i2] = sig[i2][i1] = x - pn[:, :, :, j] if i1 == i2 else x
                for c in range(d):
                    acc = 0
                    for k in range(d):
                        acc = acc + torch.bmm((dN[:, :, :, k] * dO[:, :, None]).transpose(1, 2), sig[k][c])
                    J[:, :, c, :, j] = acc
            A = J.abs()
            el = m.el[r].reshape(-1)
            rs = A.sum(dim=(3, 4))
            for c in range(d):
                rows[c].index_add_(0, el, rs[:, :, c].reshape(-1))
                diag[c].index_add_(0, el, torch.diagonal(A[:, :, c, :, c], dim1=1, dim2=2).reshape(-1))
        return rows, diag

    def solve(self, v, P, bc, eps, check, max_iter, rel_drop=1e-2, cfl=0.98, cf=0.9, thermal=None):
        """The Powell–Hestenes / Chebyshev iteration; returns v, P and the iterations done."""
        d, nn = self.dim, self.m.nn
        bc = [(torch.as_tensor(n, device="cuda"), torch.as_tensor(x, device="cuda")) for n, x in bc]
        v, P = [x.clone() for x in v], P.clone()
        rate = [torch.zeros(nn, device="cuda", dtype=F64) for _ in range(d)]
        plus = lambda x: x + (np.nextafter(abs(x), np.inf) - abs(x))
        norm = lambda x: float(torch.linalg.vector_norm(x))

        def masked(R):
            for c in range(d):
                R[c][bc[c][0]] = 0.0
            return R

        def diagnostics():
            rows, PC = self.jacobian(v, P)
            return PC, [float((rows[c] / PC[c]).max()) for c in range(d)]

        PC, lmax = diagnostics()
        step = [_chebyshev(2 / math.sqrt(x) * cfl, 0.0, cf) for x in lmax]
        err, err_min, it, ph = 2 * eps, math.inf, 0, 0
        hot = thermal is None
        v0 = p0 = v00 = 1.0
        R = None
        while ph < 1000:
            ph += 1
            R, RP, _ = self.residual(v, P, pnum=False)
            R = masked(R)
            eP = norm(RP / self.MP.reshape(-1)) / math.sqrt(RP.numel())
            ev = max(norm(x) for x in R) / (2 * math.sqrt(nn))
            if ph == 1:
                p0, v0 = plus(eP), plus(ev)
            elif ph == 2:
                p0 = plus(eP)
            err = min(max(ev, eP), max(ev / v0, eP / p0))
            if err < eps and hot:
                break
            if err > err_min * 1.05:
                rel_drop = max(rel_drop * 0.1, 1e-3)
            err_min = min(err_min, err)
            target = err * rel_drop
            while err > target or not hot:
                it += 1
                last = R
                if thermal is not None:
                    hot = thermal.step(self, v, P)
                R, RP, Pn = self.residual(v, P)
                R = masked(R)
                for c in range(d):
                    rate[c] = step[c][1] * rate[c] + R[c] / PC[c]
                    rate[c][bc[c][0]] = 0.0
                    v[c] = v[c] - step[c][0] * rate[c]
                    v[c][bc[c][0]] = bc[c][1]
                if it % check == 0:
                    ev = max(norm(x) for x in R) / (2 * math.sqrt(nn))
                    if it == check:
                        v00 = plus(ev)
                    err = ev if ev <= eps else max(ev / v00, ev)
                    lmin = []
                    for c in range(d):
                        sr = step[c][0] * rate[c]
                        den = float((sr * sr).sum())
                        lmin.append(abs(float((sr * (R[c] - last[c]) / PC[c]).sum())) / den if den else 0.0)
                    if self.pl is not None:
                        PC, lmax = diagnostics()
                    step = [_chebyshev(2 / math.sqrt(x) * cfl, y, cf) for x, y in zip(lmax, lmin)]
                if it > max_iter:
                    break
            P = P + (self.gP * RP.view_as(self.gP) / self.MP).reshape(-1)
            if it > max_iter:
                break
        return v, P, it


def _directional(f, x, dx):
    """Derivative of the list f(x) along dx (both nested lists of tensors)."""
    flat, tang = sum(x, []), sum(dx, [])
    d = len(x)
    g = lambda *a: tuple(f([list(a[i * d:(i + 1) * d]) for i in range(d)]))
    return torch.func.jvp(g, tuple(flat), tuple(tang))[1]


def _chebyshev(dtau, lmin, cf):
    c = 2 * math.sqrt(lmin) * cf
    return 2 * dtau * dtau / (2 + c * dtau), (2 - c * dtau) / (2 + c * dtau)


class _Thermal:
    """Heat-diffusion residual, its Jacobian diagnostics and DR steps."""

    def __init__(self, m, mat, phase_nodes, T, T0, P, source, bc, dt, Tref, cfl=0.98, cf=0.9, eps=1e-6):
        self.m, self.dt, self.Tref, self.cfl, self.cf, self.eps = m, dt, Tref, cfl, cf, eps
        ph = torch.as_tensor(phase_nodes, device="cuda")[m.el]
        at = lambda vals: torch.as_tensor(np.asarray(vals, dtype=np.float64), device="cuda")[ph] @ m.t.N.T
        self.k, self.Cp, self.rho0, self.alpha = at(mat["k"]), at(mat["Cp"]), at(mat["rho0"]), at(mat["alpha"])
        self.beta = at([1.0 / x for x in mat["K"]])
        dev = lambda x: torch.as_tensor(x, device="cuda", dtype=F64)
        self.T, self.T0q = dev(T).clone(), m.value(dev(T0))
        self.T0 = dev(T0)
        self.Pq, self.s = m.value(dev(P)), m.value(dev(source))
        self.bc = (torch.as_tensor(bc[0], device="cuda"), dev(bc[1]))
        self.rate, self.R = torch.zeros_like(self.T), torch.zeros_like(self.T)
        self.a = self.b = self.first = 0.0
        self.it, self.phi, self.lmax = 0, None, 0.0

    def assemble(self, jac):
        m, t = self.m, self.m.t
        Tq, gT = m.value(self.T), m.gradient(self.T)
        rho = self.rho0 * (1 - self.alpha * (Tq - self.Tref) + self.beta * self.Pq)
        dtrc = self.dt / (rho * self.Cp)
        heat = self.s + (self.phi if self.phi is not None else 0.0)
        self.R = m.scatter([-dtrc * self.k * x for x in gT], self.T0q - Tq + dtrc * heat)
        if not jac:
            return
        rows, diag = torch.zeros_like(self.T), torch.zeros_like(self.T)
        cfac = dtrc * self.alpha * self.rho0 / rho
        for s0 in range(0, m.ne, 4096):
            r = slice(s0, min(s0 + 4096, m.ne))
            dN, dO, N = m.physical(r), m.dO[r], t.N
            KT = sum(dN[:, :, :, k] * gT[k][r][:, :, None] for k in range(m.dim))      # e q i
            left = N[None] * (-1.0 + (cfac * heat)[r])[:, :, None] - (cfac * self.k)[r][:, :, None] * KT
            J = torch.bmm((left * dO[:, :, None]).transpose(1, 2), N[None].expand(left.shape[0], -1, -1))
            w = (dtrc * self.k)[r] * dO
            for k in range(m.dim):
                J = J - torch.bmm((dN[:, :, :, k] * w[:, :, None]).transpose(1, 2), dN[:, :, :, k])
            A = J.abs()
            el = m.el[r].reshape(-1)
            rows.index_add_(0, el, A.sum(dim=2).reshape(-1))
            diag.index_add_(0, el, torch.diagonal(A, dim1=1, dim2=2).reshape(-1))
        self.PC, self.lmax = diag, float((rows / diag).max())

    def advance(self, check):
        """One DR step; on a check the error and the next step's coefficients."""
        self.it += 1
        look = self.it == 1 or self.it % check == 0
        last = self.R
        self.assemble(look)
        r = self.R / self.PC + self.b * self.rate
        self.R[self.bc[0]] = 0.0
        r[self.bc[0]] = 0.0
        self.rate = r
        self.T = self.T + self.a * r
        self.T[self.bc[0]] = self.bc[1]
        if not look:
            return None
        dtau = 2 / math.sqrt(self.lmax) * self.cfl
        nr = float(torch.linalg.vector_norm(self.R))
        if self.it == 1:
            self.first = nr
        sr = dtau * self.rate
        den = float((sr * sr).sum())
        lmin = 0.0 if self.it == 1 or den == 0 else abs(float((sr * (self.R - last) / self.PC).sum())) / den
        self.a, self.b = _chebyshev(dtau, lmin, self.cf)
        return nr / self.first


class _Coupling:
    """The thermal step inside the Stokes loop: temperature to the pressure nodes, shear heat back."""

    def __init__(self, thermal, stokes, check, v, P):
        self.th, self.check, self.done = thermal, check, False
        self.pn = stokes.m.el[:, _PNODES[3]]
        stokes.T, stokes.T0 = thermal.T[self.pn], thermal.T0[self.pn]
        thermal.phi = stokes.heating(v, P)

    def step(self, stokes, v, P):
        err = self.th.advance(self.check)
        stokes.T = self.th.T[self.pn]
        if err is not None:
            self.done = err < self.th.eps
            self.th.phi = stokes.heating(v, P)
        return self.done


def _images(case, seed):
    """BF16 network inputs (8 of 16 channels used) and FP32 targets, smooth fields plus noise."""
    B, H, W = case["images"], case["height"], case["width"]
    g = _gen(seed)
    low = torch.randn(B, 11, 9, 9, generator=g, device="cuda")
    f = torch.nn.functional.interpolate(low, size=(H, W), mode="bilinear", align_corners=True)
    f = f.permute(0, 2, 3, 1) + 0.1 * torch.randn(B, H, W, 11, generator=g, device="cuda")
    x = torch.zeros(B, H, W, 16, device="cuda", dtype=torch.bfloat16)
    x[..., :8] = f[..., :8].to(torch.bfloat16)
    return x.reshape(-1).contiguous(), f[..., 8:].float().reshape(-1).contiguous()


def _network_exact(case, seed):
    B, H, W = case["images"], case["height"], case["width"]
    g = torch.Generator().manual_seed(int(seed))
    chans = [16] + [32] * 5 + [16]
    ws, bs = [], []
    for i in range(6):
        ci, co = chans[i], chans[i + 1]
        bound = math.sqrt(6.0 / (9 * ci)) * (0.1 if i == 5 else 1.0)
        w = (torch.rand(co, 9 * ci, generator=g) * 2 - 1) * bound
        w = w.cuda().to(torch.bfloat16).double()          # the network multiplies by its BF16 copies
        ws.append(w.view(co, 3, 3, ci).permute(0, 3, 1, 2).contiguous().requires_grad_())
        bs.append(torch.zeros(co, device="cuda", dtype=F64, requires_grad=True))
    x, target = _images(case, seed)
    loss, out = 0.0, []
    # image by image: the 64-bit activations of all eight need not be held together
    for b in range(B):
        h = x.view(B, H, W, 16)[b:b + 1].double().permute(0, 3, 1, 2)
        for i in range(6):
            h = torch.nn.functional.conv2d(h, ws[i], bs[i], padding=1)
            if i < 5:
                h = torch.relu(h)
        if not case["train"]:
            out.append(h.detach().permute(0, 2, 3, 1).reshape(-1))
            continue
        diff = h[:, :3] - target.view(B, H, W, 3)[b:b + 1].double().permute(0, 3, 1, 2)
        part = (diff * diff).sum() / (B * H * W)
        part.backward()
        loss += float(part.detach())
    if not case["train"]:
        return {"out": torch.cat(out)}
    gw = []
    for w in ws:
        co, ci = w.shape[:2]
        full = torch.zeros(co, 9 * ci + 8, device="cuda", dtype=F64)
        full[:, :9 * ci] = w.grad.permute(0, 2, 3, 1).reshape(co, 9 * ci)
        gw.append(full)
    return {"loss": loss, "gw": gw, "gb": [b.grad for b in bs]}


def _cell_pressure_exact(case, seed):
    inp = _block(case, seed)
    m = _Mesh(inp["box"])
    t, ne, mat = m.t, m.ne, inp["mat"]
    ph = torch.as_tensor(inp["phase"], device="cuda")
    eta = torch.as_tensor(mat["eta"], device="cuda", dtype=F64)[ph][:, None]
    rho = torch.as_tensor(mat["rho0"], device="cuda", dtype=F64)[ph][:, None].expand(ne, t.nq)
    modes = torch.cat([torch.ones(t.nq, 1, device="cuda", dtype=F64), t.x], dim=1)      # q m
    M = m.dO @ (modes * modes)
    diag = torch.zeros(3, m.nn, device="cuda", dtype=F64)
    for s0 in range(0, ne, 8192):
        r = slice(s0, min(s0 + 8192, ne))
        dN = m.physical(r)
        n2 = (dN * dN).sum(dim=-1)
        w = (m.dO * eta)[r][:, :, None]
        for c in range(3):
            diag[c].index_add_(0, m.el[r].reshape(-1), ((n2 + dN[..., c] ** 2 / 3) * w).sum(dim=1).reshape(-1))
    bc = [torch.as_tensor(n, device="cuda") for n, _ in inp["bc"]]
    v = [torch.zeros(m.nn, device="cuda", dtype=F64) for _ in range(3)]
    P = torch.zeros(ne, 4, device="cuda", dtype=F64)
    for it in range(1, case["iterations"] + 1):
        gr = [m.gradient(u) for u in v]
        RP = -((gr[0][0] + gr[1][1] + gr[2][2]) * m.dO) @ modes
        P = P + 0.2 * RP / M
        P[:, 0] -= (P[:, 0] * M[:, 0]).sum() / M[:, 0].sum()
        tr = (gr[0][0] + gr[1][1] + gr[2][2]) / 3
        Pq = P @ modes.T
        err = 0.0
        for c in range(3):
            s = [eta * (gr[c][k] + gr[k][c]) for k in range(3)]
            s[c] = s[c] - 2 * eta * tr - Pq
            R = m.scatter(s, -rho * mat["g"][c] if mat["g"][c] else None)
            R[bc[c]] = 0.0
            v[c] = v[c] - 0.6 * R / diag[c]
            if it % 100 == 0:
                err = max(err, float(torch.linalg.vector_norm(R)))
        if it % 100 == 0 and max(err, float(torch.linalg.vector_norm(RP))) < 1e-8:
            break
    return {"v": v, "P": P.reshape(-1), "iterations": it}


def _adjoint_exact(case, seed):
    inp = _hot(case, seed)
    s = _Stokes(inp)
    s.scaling()
    v = [x.clone().requires_grad_() for x in inp["v"]]
    P = inp["P"].clone().requires_grad_()
    eta = s.eta.clone().requires_grad_()
    s.eta = eta
    Rv, RP, _ = s.residual(v, P)
    s.eta = eta.detach()
    with torch.no_grad():
        rows, PC = s.jacobian([x.detach() for x in v], P.detach())
    nn, nP, eps, cfl, cf = s.m.nn, P.numel(), 1e-6, 0.98, 0.9
    bc = [torch.as_tensor(n, device="cuda") for n, _ in inp["bc"]]
    lv = [torch.zeros(nn, device="cuda", dtype=F64) for _ in range(3)]
    lP = torch.zeros(nP, device="cuda", dtype=F64)
    rate = [torch.zeros_like(x) for x in lv]
    dtau = [2 / math.sqrt(float((rows[c] / PC[c]).max())) * cfl for c in range(3)]
    step = [_chebyshev(x, 0.0, cf) for x in dtau]
    plus = lambda x: x + (np.nextafter(abs(x), np.inf) - abs(x))

    def assemble():
        gr = torch.autograd.grad([*Rv, RP], [*v, P], [*lv, lP], retain_graph=True)
        R = [gr[c] + inp["objective"][c] for c in range(3)]
        for c in range(3):
            R[c][bc[c]] = 0.0
        return R, gr[3]

    verr = lambda R: max(float(torch.linalg.vector_norm(x)) for x in R) / math.sqrt(nn)
    it, v0, p0 = 0, 1.0, 1.0
    for ph in range(1, 101):
        R, dP = assemble()
        ev, ep = verr(R), float(torch.linalg.vector_norm(dP)) / math.sqrt(nP)
        if ph == 1:
            v0, p0 = plus(ev), plus(ep)
        if max(min(ev, ev / v0), min(ep, ep / p0)) < eps:
            break
        target = max(ev * 0.1, eps)
        while ev > target and it < case["iterations"]:
            it += 1
            last = R
            for c in range(3):
                rate[c] = step[c][1] * rate[c] + R[c] / PC[c]
                rate[c][bc[c]] = 0.0
                lv[c] = lv[c] - step[c][0] * rate[c]
            R, dP = assemble()
            if it % 50 == 0:
                ev = verr(R)
                for c in range(3):
                    sr = step[c][0] * rate[c]
                    den = float((sr * sr).sum())
                    lmin = abs(float((sr * (R[c] - last[c]) / PC[c]).sum())) / den if den else 0.0
                    step[c] = _chebyshev(dtau[c], lmin, cf)
        lP = lP + s.gP.reshape(-1) * dP / s.MP.reshape(-1)
        if it >= case["iterations"]:
            break
    # the sensitivity is that of the momentum residual's stress at the fixed pressures
    g = torch.autograd.grad([*Rv], [eta], [*lv], retain_graph=False)[0]
    return {"lam_v": lv, "lam_P": lP, "sensitivity": g.reshape(-1), "iterations": it}


def exact(case, seed):
    kind = case["kind"]
    if kind == "network":
        return _network_exact(case, seed)
    if kind == "cell_pressure":
        return _cell_pressure_exact(case, seed)
    if kind == "adjoint":
        return _adjoint_exact(case, seed)
    inp = _INPUTS[kind](case, seed)
    if kind == "thermal":
        th = _Thermal(_Mesh(inp["box"]), inp["mat"], inp["phase_nodes"], inp["T"], inp["T"], inp["P"], inp["source"],
                      inp["bc"], inp["dt"], inp["Tref"])
        for it in range(1, case["iterations"] + 1):
            err = th.advance(50)
            if err is not None and err < 1e-12:
                break
        return {"T": th.T, "R": th.R, "iterations": it}
    s = _Stokes(inp)
    v = [torch.as_tensor(x, device="cuda", dtype=F64) for x in inp["v"]]
    P = inp["P"] if "P" in inp else torch.zeros(s.m.ne * s.box.np, device="cuda", dtype=F64)
    if kind == "residual":
        Rv, RP, Pn = s.residual(v, P)
        return {"Rv": Rv, "RP": RP, "Pnum": Pn}
    if kind == "jacobian":
        rows, diag = s.jacobian(v, P)
        return {"rows": list(rows), "diag": list(diag)}
    s.scaling()
    if kind == "coupled":
        box = inp["box"]
        T = _nodal_T(box, seed)
        th = _Thermal(s.m, dict(k=[1.0], Cp=[1.0], rho0=[1.0], alpha=[0.1], K=[math.inf]),
                      np.zeros(box.nnodes, dtype=np.int64), T, T, np.zeros(box.nnodes), np.zeros(box.nnodes),
                      _thermal_walls(box), inp["dt"], 0.0)
        cp = _Coupling(th, s, case["check"], v, P)
        v, P, it = s.solve(v, P, inp["bc"], 1e-8, case["check"], case["iterations"], thermal=cp)
        return {"v": v, "P": P, "T": th.T, "iterations": it}
    v, P, it = s.solve(v, P, inp["bc"], 1e-8, case["check"], case["iterations"])
    return {"v": v, "P": P, "iterations": it}
