"""Performance cases of the FEM + SIMP path, through the entry points a host program calls.

A case is a dict of plain values; ``prepare`` makes what a host program holds before the call (a FeModel and its
options, a resident problem with its filter, a density field), ``run`` is one pass through the public entry
points, ``exact`` the same results in plain 64-bit torch arithmetic.

kinds
  static  StaticAnalysis.run: one analysis of a host model (upload, set-up, solve, reactions, von Mises, results)
  simp    TopologyOptimizer.run: a whole optimisation of a few SIMP iterations from a host model
  many    TopologyOptimizer.run_many: uneven optimisations side by side, their solves packed
  update  the kernel-level calls of a host-driven design update on a resident problem: densities, filter,
          product with K, sensitivities, adjoint filter, OC
  mesh    export of a density field: SurfaceNetsExtractor.extract and TaubinSmoother.smooth
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mycel_b200 import api
from mycel_b200 import workloads as W
from mycel_b200.model import FeMaterial, FeModel, GridSpec, LoadCase, OptimizerOptions, StaticAnalysisOptions, SurfacePatch

MG = ("mg", "mixed-mg")


def listed():
    static = dict(kind="static", h=1.0, nu=0.3, emin=1e-9, loads=1)
    simp = dict(kind="simp", h=1.0, nu=0.3, emin=1e-9, loads=1, apart=False, heaviside=False, start="uniform")
    return [
        # the reference's small test cantilever analysed in the default (plain FP64) form: latency and set-up
        dict(static, name="static-fp64-30x10x4", shape="cantilever", nx=30, ny=10, nz=4, precision="fp64", tol=1e-6,
             emin=1e-6),
        # the static benchmark: a carved part with graded densities, the drop-in form, to 1e-8
        dict(static, name="static-fp64-96x48x24", shape="carved", nx=96, ny=48, nz=24, precision="fp64", tol=1e-8),
        # the reference's scaling benchmark shape (5d x d x d, its first published size) in the FP64 multigrid form
        dict(static, name="static-mg-110x22x22", shape="cantilever", nx=110, ny=22, nz=22, precision="mg", tol=1e-6,
             emin=1e-6),
        # a ragged carved part in the fast FP64 form (Jacobi)
        dict(static, name="static-fp64f-61x37x23", shape="carved", nx=61, ny=37, nz=23, precision="fp64f", tol=1e-8,
             h=2.5, nu=0.28),
        # analysis of the largest single-GPU grid in the fast form, results read back whole
        dict(static, name="static-mixed-mg-192x96x96", shape="bridge", nx=192, ny=96, nz=96, precision="mixed-mg",
             tol=1e-8),
        # the plain FP64 SIMP cantilever (8,000 elements, rmin 1.5, tolerance 1e-8): the default optimisation form
        dict(simp, name="simp-fp64-40x20x10", shape="cantilever", nx=40, ny=20, nz=10, precision="fp64", tol=1e-8,
             iterations=6, volfrac=0.3, rmin=1.5),
        # the headline workload: the 192x96x96 bridge (volfrac 0.15, rmin 2.5, tolerance 1e-6) in its fastest form
        dict(simp, name="simp-mixed-mg-192x96x96", shape="bridge", nx=192, ny=96, nz=96, precision="mixed-mg",
             tol=1e-6, iterations=8, volfrac=0.15, rmin=2.5),
        # a served job: a carved part of odd sizes, resumed from a snapshot's densities
        dict(simp, name="simp-mixed-mg-85x53x27", shape="carved", nx=85, ny=53, nz=27, precision="mixed-mg", tol=1e-8,
             iterations=6, volfrac=0.3, rmin=2.2, start="random"),
        # a batched instance: four load cases kept apart on one stiffness
        dict(simp, name="simp-mixed-mg-64x32x40-4cases", shape="cantilever", nx=64, ny=32, nz=40,
             precision="mixed-mg", tol=1e-8, iterations=4, volfrac=0.25, rmin=1.8, loads=4, apart=True),
        # many uneven optimisations side by side (the batched workload at reduced count and iterations)
        dict(kind="many", name="many-mixed-mg-8", count=8, batch=7, scale=0.5, iterations=4, precision="mixed-mg", tol=1e-8),
        # a host-driven design update at the level-1 size of the bridge, host arrays in and out
        dict(kind="update", name="update-96x48x48", nx=96, ny=48, nz=48, rmin=2.5, volfrac=0.3, h=1.0, nu=0.3,
             emin=1e-9),
        # export of a design on the largest grid
        dict(kind="mesh", name="mesh-192x96x96", nx=192, ny=96, nz=96, waves=9, pattern=1, smooth=3),
    ]


def _sizes(rng, lo, hi):
    """nx >= ny, nz of odd proportions with about a log-uniform number of elements in [lo, hi]."""
    ne = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(0.3, 1.0), rng.uniform(0.25, 1.0)
    nx = max(8, round((ne / (a * b)) ** (1 / 3)))
    ny = max(4, round(a * nx))
    return nx, ny, max(4, round(ne / (nx * ny)))


def draw(rng):
    kind = rng.choice(["static", "static", "static", "simp", "simp", "simp", "many", "update", "mesh"])
    h, nu, emin = rng.choice([1.0, 1.0, 0.5, 2.5]), rng.choice([0.3, 0.3, 0.28]), rng.choice([1e-9, 1e-9, 1e-6])
    if kind == "static":
        precision = rng.choice(["fp64", "fp64", "fp64f", "mg", "mixed-mg", "mixed-mg"])
        nx, ny, nz = _sizes(rng, 1200, {"fp64": 110_000, "fp64f": 150_000}.get(precision, 1_700_000))
        return dict(kind=kind, shape=rng.choice(["cantilever", "carved"]) if nx * ny * nz < 200_000 else "bridge",
                    nx=nx, ny=ny, nz=nz, precision=precision, tol=rng.choice([1e-6, 1e-8]), h=h, nu=nu, emin=emin,
                    loads=rng.randint(1, 3))
    if kind == "simp":
        precision = rng.choice(["fp64", "mixed-mg", "mixed-mg", "mixed-mg"])
        nx, ny, nz = _sizes(rng, 1200, 12_000 if precision == "fp64" else 400_000)
        loads = rng.randint(1, 4)
        return dict(kind=kind, shape=rng.choice(["cantilever", "carved"]) if nx * ny * nz < 200_000 else "bridge",
                    nx=nx, ny=ny, nz=nz, precision=precision, tol=1e-8, h=h, nu=nu, emin=emin,
                    iterations=rng.randint(2, 4), volfrac=round(rng.uniform(0.1, 0.4), 3),
                    rmin=round(rng.uniform(1.2, 3.0), 2), loads=loads, apart=loads > 1 and rng.random() < 0.5,
                    heaviside=rng.random() < 0.2, start=rng.choice(["uniform", "random"]))
    if kind == "many":
        return dict(kind=kind, count=rng.randint(3, 8), batch=rng.randint(1, 10_000), scale=round(rng.uniform(0.5, 0.8), 3),
                    iterations=rng.randint(2, 4), precision="mixed-mg", tol=1e-8)
    nx, ny, nz = _sizes(rng, 2000, 1_700_000 if kind == "mesh" else 400_000)
    if kind == "update":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, rmin=round(rng.uniform(1.2, 3.0), 2),
                    volfrac=round(rng.uniform(0.1, 0.4), 3), h=h, nu=nu, emin=emin)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, waves=rng.randint(3, 12), pattern=rng.randint(1, 10_000),
                smooth=rng.randint(1, 5))


# ---- inputs -----------------------------------------------------------------------------------------------
def _unit(rng):
    v = rng.normal(size=3)
    return v / np.linalg.norm(v)


def _face_loads(rng, g, node_act, count):
    """Load cases of random unit direction on 4 x 4 node patches of the active x = nx face."""
    out = []
    for _ in range(count):
        j0, k0 = int(rng.integers(0, max(1, g.ny - 2))), int(rng.integers(0, max(1, g.nz - 2)))
        face = [(j, k) for k in range(g.nz + 1) for j in range(g.ny + 1) if node_act[k, j, g.nx]]
        patch = [(j, k) for j, k in face if j0 <= j < j0 + 4 and k0 <= k < k0 + 4] or face
        nodes = [g.node_index(g.nx, j, k) for j, k in patch]
        out.append(LoadCase(SurfacePatch(nodes, np.ones(len(nodes))), tuple(float(v) for v in _unit(rng))))
    return out


def _model(case, seed):
    """The model of a static or simp case: domain, supports and loads of its shape, loads seeded."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mat = FeMaterial(1.0, case["nu"], case["emin"])
    if case["shape"] == "bridge":
        s = max(2, min(8, nx // 8, ny // 6))
        m = W.bridge(nx, ny, nz, support=s, load_patch=2 * s)
        v = 0.3 * _unit(rng) + np.array([0.0, 0.0, -1.0])  # mostly downwards
        loads = [LoadCase(m.loads[0].patch, tuple(float(x) for x in v))]
        for _ in range(case["loads"] - 1):
            loads.append(LoadCase(m.loads[0].patch, tuple(float(x) for x in _unit(rng))))
        domain, fixed = m.domain, m.fixed_dofs
    else:
        m = (W.served_job(nx, ny, nz, 1, int(rng.integers(2**31)))[0] if case["shape"] == "carved"
             else W.cantilever(nx, ny, nz))
        domain, fixed = m.domain, m.fixed_dofs
        loads = _face_loads(rng, m.grid, m.active_nodes_mask().reshape(nz + 1, ny + 1, nx + 1), case["loads"])
    dens = rng.uniform(0.1, 1.0, nx * ny * nz) if case["kind"] == "static" else None
    return FeModel(GridSpec(nx, ny, nz, case["h"]), domain, mat, fixed, loads, element_density=dens)


def _simp_options(case, seed):
    ne = case["nx"] * case["ny"] * case["nz"]
    rho = None
    if case["start"] == "random":  # resumed from a snapshot: densities about the volume fraction
        rho = np.random.default_rng(seed + 1).uniform(0.5, 1.5, ne) * case["volfrac"]
    return OptimizerOptions(
        volume_fraction=case["volfrac"], filter_radius_mm=case["rmin"] * case["h"], penal=3.0, move_limit=0.2,
        max_iterations=case["iterations"], solver_tolerance_initial=case["tol"], solver_tolerance_final=case["tol"],
        solver_max_iterations=20000, enable_heaviside=case["heaviside"], precision=case["precision"],
        separate_load_cases=case["apart"], initial_density=None if rho is None else rho.astype(np.float32))


def _waves(n, count, seed):
    """A smooth field of unit size: a few plane waves of random direction, wavelength and phase."""
    g = torch.Generator().manual_seed(int(seed) % (1 << 31))
    z, y, x = (torch.arange(k, device="cuda", dtype=torch.float32) / max(n) for k in n)
    f = torch.zeros(n, device="cuda")
    for _ in range(count):
        k = (torch.randn(3, generator=g) * 14).tolist()
        ph = float(torch.rand(1, generator=g)) * 6.2832
        f += torch.cos(k[0] * z[:, None, None] + k[1] * y[None, :, None] + k[2] * x[None, None, :] + ph)
    return f / math.sqrt(count)


def _field(case, seed):
    """A smooth density in [0, 1]: the solid part (above 0.5) is the case's pattern, the densities are the seed's."""
    n = [case["nz"], case["ny"], case["nx"]]
    f = _waves(n, case["waves"], case["pattern"])
    f = torch.where(f < 0, f.clamp_max(-1e-3), f.clamp_min(1e-3))
    return torch.sigmoid(4 * f * torch.exp(0.3 * _waves(n, 3, seed).clamp(-2, 2))).cpu().numpy().reshape(-1)


def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind == "static":
        return dict(kind=kind, model=_model(case, seed),
                    options=StaticAnalysisOptions(tolerance=case["tol"], max_iterations=20000,
                                                  precision=case["precision"]))
    if kind == "simp":
        return dict(kind=kind, model=_model(case, seed), options=_simp_options(case, seed))
    if kind == "many":
        rng = np.random.default_rng(seed)
        jobs = W.batched_instances(count=case["count"], seed=case["batch"], scale=case["scale"])
        models = [FeModel(m.grid, m.domain, m.material, m.fixed_dofs,
                          [LoadCase(lc.patch, tuple(float(v) for v in _unit(rng))) for lc in m.loads])
                  for m in (j.model for j in jobs)]
        return dict(kind=kind, models=models,
                    options=[j.options.replace(max_iterations=case["iterations"], precision=case["precision"],
                                               solver_tolerance_initial=case["tol"],
                                               solver_tolerance_final=case["tol"]) for j in jobs])
    if kind == "update":
        rng = np.random.default_rng(seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        m = W.cantilever(nx, ny, nz, case["h"], e0=1.0, nu=case["nu"], emin_ratio=case["emin"], force=-1.0)
        p = api.Problem(m)
        f = api.DensityFilter(p, case["rmin"])
        n = np.arange(m.total_nodes)
        i, j, k = n % (nx + 1), n // (nx + 1) % (ny + 1), n // ((nx + 1) * (ny + 1))
        w = rng.uniform(0.5, 3.0, (3, 3))  # a smooth displacement field of the size of the part's deflection
        u = np.stack([(i / nx) ** 2 * np.cos(w[c, 0] * i / nx + w[c, 1] * j / ny + w[c, 2] * k / nz)
                      for c in range(3)], axis=1).reshape(-1)
        return dict(kind=kind, problem=p, filter=f, s=f.s, rho=rng.uniform(0.01, 1.0, m.active_element_count), u=u,
                    volfrac=case["volfrac"])
    return dict(kind=kind, grid=GridSpec(case["nx"], case["ny"], case["nz"]), density=_field(case, seed),
                smooth=case["smooth"])


# ---- one pass ---------------------------------------------------------------------------------------------
def _optimised(r):
    return dict(u=r.final_displacements, physical=r.final_physical_density, design=r.final_design_density,
                compliance=np.array([s.compliance for s in r.snapshots]),
                volume=np.array([s.volume_fraction for s in r.snapshots]))


def run(state):
    kind = state["kind"]
    if kind == "static":
        r = api.StaticAnalysis.run(state["model"], state["options"])
        return dict(u=r.u, compliance=r.compliance, max_displacement=r.max_displacement, reactions=r.reactions,
                    von_mises=r.von_mises_per_element)
    if kind == "simp":
        return _optimised(api.TopologyOptimizer.run(state["model"], state["options"]))
    if kind == "many":
        return [_optimised(r) for r in api.TopologyOptimizer.run_many(state["models"], state["options"])]
    if kind == "update":
        p, f = state["problem"], state["filter"]
        phys = f.apply(state["rho"])
        p.update_densities(phys, 3.0)  # every element of the box is active
        ku = p.apply_k(state["u"])
        dc = f.adjoint(p.sensitivities(state["u"], phys, 3.0))
        rho, lam = api.oc_update(state["rho"], dc, state["s"], None, state["volfrac"])
        return dict(physical=phys, ku=ku, dc=dc, rho=rho, lam=lam)
    mesh = api.SurfaceNetsExtractor.extract(state["grid"], state["density"], 0.5)
    smooth = api.TaubinSmoother.smooth(mesh, state["smooth"])
    return dict(positions=mesh.positions, indices=mesh.indices, smoothed=smooth.positions)


# ---- what a pass cannot do without ------------------------------------------------------------------------
def work(case):
    """Inputs read and results written once, and for each solve the products with K that its form needs (x read,
    y and the search direction written per product; Jacobi counts grow with the longest axis, multigrid's do
    not)."""
    if case["kind"] == "many":
        one = dict(case, kind="simp", nx=round(76 * case["scale"]), ny=round(38 * case["scale"]),
                   nz=max(2, round(36 * case["scale"])), loads=1, apart=False)
        w = work(one)
        return {k: v * case["count"] for k, v in w.items()}
    ne = case["nx"] * case["ny"] * case["nz"]
    nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if case["kind"] == "mesh":
        surface = 2 * case["waves"] * (case["nx"] * case["ny"] + case["ny"] * case["nz"] + case["nx"] * case["nz"])
        return dict(bytes=4 * ne + 48 * surface, flops=60 * surface * (1 + case["smooth"]))
    if case["kind"] == "update":
        terms = 4 / 3 * math.pi * max(1.5, case["rmin"]) ** 3
        return dict(bytes=8 * (9 * ne + 9 * nn), flops=ne * (4 * terms + 2 * 1152 + 400))
    decades = -math.log10(case["tol"])
    fp64 = case["precision"] in ("fp64", "fp64f")
    products = (1.2 * max(case["nx"], case["ny"], case["nz"]) * decades) if fp64 else 12 * decades
    solves = case.get("iterations", 1) * (case["loads"] if case.get("apart") else 1)
    per = 1152 if case["precision"] == "fp64" else 190
    size = 4 if case["precision"] == "mixed-mg" else 8
    io = 9 * ne + 24 * nn + (24 * nn + 8 * ne if case["kind"] == "static" else 8 * ne)
    return dict(bytes=io + solves * products * (9 * size * nn), flops=solves * products * per * ne)


# ---- the same results in 64 bits --------------------------------------------------------------------------
class _Fem:
    """Hex8 voxels in plain torch FP64: K u, Jacobi-PCG, energies, centroid stresses."""

    LOCAL = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]

    def __init__(self, model):
        g = self.g = model.grid
        h, nu = float(np.float32(g.h)), model.material.nu
        self.h = h
        self.d = np.zeros((6, 6))
        c = 1.0 / ((1 + nu) * (1 - 2 * nu))
        self.d[:3, :3] = c * nu
        self.d[np.arange(3), np.arange(3)] = c * (1 - nu)
        self.d[np.arange(3, 6), np.arange(3, 6)] = 0.5 / (1 + nu)
        ke = np.zeros((24, 24))
        q = 1 / math.sqrt(3)
        for x in (-q, q):
            for y in (-q, q):
                for z in (-q, q):
                    b = self.strain(x, y, z)
                    ke += b.T @ self.d @ b / 8
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.ke = self.t(ke * h)
        self.dom = self.t(model.domain.reshape(g.nz, g.ny, g.nx) != 0)
        e = torch.nonzero(self.dom.reshape(-1)).reshape(-1)
        ix, iy, iz = e % g.nx, e // g.nx % g.ny, e // (g.nx * g.ny)
        nodes = torch.stack([(ix + a) + (g.nx + 1) * ((iy + b) + (g.ny + 1) * (iz + c)) for a, b, c in self.LOCAL], 1)
        self.active = e
        self.dofs = (3 * nodes[:, :, None] + torch.arange(3, device=dev)).reshape(-1, 24)
        free = torch.zeros(g.total_dofs, dtype=torch.bool, device=dev)
        free[self.dofs.reshape(-1)] = True
        free[self.t(model.fixed_dofs.astype(np.int64))] = False
        self.free = free
        self.fixed = self.t(np.unique(model.fixed_dofs).astype(np.int64))
        self.cases = []
        for lc in model.loads:
            f = torch.zeros(g.total_dofs, dtype=torch.float64, device=dev)
            w = self.t(lc.patch.node_area / lc.patch.node_area.sum())
            for k in range(3):
                f.index_add_(0, self.t(3 * lc.patch.nodes.astype(np.int64) + k), w * lc.total_force[k])
            self.cases.append(f)
        self.e0, self.emin = model.material.e0, model.material.emin

    def strain(self, x, y, z):
        b = np.zeros((6, 24))
        for a, (i, j, k) in enumerate(self.LOCAL):
            s, t, r = 2 * i - 1, 2 * j - 1, 2 * k - 1
            gx = s * (1 + t * y) * (1 + r * z) / 4
            gy = t * (1 + s * x) * (1 + r * z) / 4
            gz = r * (1 + s * x) * (1 + t * y) / 4
            b[0, 3 * a] = b[4, 3 * a + 2] = b[5, 3 * a + 1] = gx
            b[1, 3 * a + 1] = b[3, 3 * a + 2] = b[5, 3 * a] = gy
            b[2, 3 * a + 2] = b[3, 3 * a + 1] = b[4, 3 * a] = gz
        return b

    def young(self, rho, penal=3.0):
        return self.emin + rho.double() ** penal * (self.e0 - self.emin)

    def apply(self, e, u):
        f = (u[self.dofs] * e[:, None]) @ self.ke
        return torch.zeros_like(u).index_add_(0, self.dofs.reshape(-1), f.reshape(-1))

    def solve(self, e, f, tol=1e-13, most=12000):
        diag = torch.zeros_like(f).index_add_(0, self.dofs.reshape(-1), (e[:, None] * self.ke.diagonal()).reshape(-1))
        inv = torch.where(self.free, 1.0 / diag.clamp_min(1e-300), 0.0)
        b = torch.where(self.free, f, 0.0)
        u, target = torch.zeros_like(b), tol * float(b.norm())
        for _ in range(3):  # restarted from the true residual
            r = torch.where(self.free, b - self.apply(e, u), 0.0)
            if float(r.norm()) <= target:
                break
            z = inv * r
            p, rz = z.clone(), r @ z
            for it in range(most):
                q = torch.where(self.free, self.apply(e, p), 0.0)
                alpha = rz / (p @ q)
                u += alpha * p
                r -= alpha * q
                if it % 25 == 0 and float(r.norm()) <= 0.5 * target:
                    break
                z = inv * r
                new = r @ z
                p = z + (new / rz) * p
                rz = new
        return u

    def energy(self, u):
        v = u[self.dofs]
        return ((v @ self.ke) * v).sum(1)

    def von_mises(self, e, u):
        s = (u[self.dofs] @ self.t(self.strain(0.0, 0.0, 0.0)).T / self.h) @ self.t(self.d).T * e[:, None]
        v = 0.5 * ((s[:, 0] - s[:, 1]) ** 2 + (s[:, 1] - s[:, 2]) ** 2 + (s[:, 2] - s[:, 0]) ** 2)
        out = torch.zeros(self.g.total_elements, dtype=torch.float64, device=u.device)
        out[self.active] = torch.sqrt(v + 3 * (s[:, 3:] ** 2).sum(1))
        return out

    def box(self, active, fill=0.0):
        out = torch.full((self.g.total_elements,), fill, dtype=torch.float64, device=active.device)
        out[self.active] = active
        return out.reshape(self.dom.shape)


class _Cone:
    """Cone filter over the active elements and its adjoint."""

    def __init__(self, fem, rmin):
        self.fem, self.r = fem, math.ceil(rmin)
        self.off = [(a, b, c, rmin - math.sqrt(a * a + b * b + c * c)) for a in range(-self.r, self.r + 1)
                    for b in range(-self.r, self.r + 1) for c in range(-self.r, self.r + 1)
                    if a * a + b * b + c * c < rmin * rmin]
        self.hs = self.spread(fem.dom.double())
        self.s = self.adjoint(torch.ones_like(fem.active, dtype=torch.float64))

    def spread(self, box):
        r, (nz, ny, nx) = self.r, box.shape
        pad = torch.nn.functional.pad(box, (r,) * 6)
        out = torch.zeros_like(box)
        for a, b, c, w in self.off:
            out += w * pad[r + a:r + a + nz, r + b:r + b + ny, r + c:r + c + nx]
        return out

    def apply(self, x):
        return (self.spread(self.fem.box(x)) / self.hs).reshape(-1)[self.fem.active]

    def adjoint(self, x):
        return self.spread(self.fem.box(x) / self.hs.clamp_min(1e-300)).reshape(-1)[self.fem.active]


def _oc(rho, dc, s, passive, volfrac, guess, move=0.2, low=1e-3):
    lo, hi = (rho - move).clamp_min(low), (rho + move).clamp_max(1.0)

    def at(lam):
        new = torch.minimum(torch.maximum(rho * torch.sqrt((-dc).clamp_min(0) / (lam * s)), lo), hi)
        new = torch.where(dc < 0, new, lo)
        return torch.where(passive, torch.ones_like(new), new)

    target = volfrac * float(s.sum())

    def volume(lam):
        return float((s * at(lam)).sum())

    l1, l2 = 0.5 * guess, 2.0 * guess
    while volume(l1) < target and l1 > 1e-50:
        l1, l2 = l1 * 0.1, l1
    while volume(l2) > target and l2 < 1e50:
        l1, l2 = l2, l2 * 10
    lam = math.sqrt(l1 * l2)
    for _ in range(60):
        lam = math.sqrt(l1 * l2)
        v = volume(lam)
        if abs(v - target) / max(target, 1e-12) <= 1e-8:
            break
        l1, l2 = (lam, l2) if v > target else (l1, lam)
        if abs(l2 - l1) <= 1e-15 * lam:
            break
    return at(lam), lam


def _exact_simp(model, o):
    fem = _Fem(model)
    g = fem.g
    flt = _Cone(fem, max(1.5, o.filter_radius_mm / fem.h))
    shell = torch.zeros_like(fem.dom)  # elements touching a supported or loaded node stay solid
    ids = np.concatenate([model.fixed_dofs // 3] + [lc.patch.nodes for lc in model.loads])
    for n in np.unique(ids):
        i, j, k = g.inverse_node_index(int(n))
        z, y, x = (slice(min(max(v - 1, 0), c - 1), min(v, c - 1) + 1) for v, c in ((k, g.nz), (j, g.ny), (i, g.nx)))
        shell[z, y, x] = True
    passive = shell.reshape(-1)[fem.active]
    if o.initial_density is None:
        rho = torch.full_like(flt.s, o.volume_fraction)
    else:
        rho = fem.t(o.initial_density.astype(np.float64))[fem.active]
    rho = torch.where(passive, torch.ones_like(rho), rho)
    lam, comp, vol, u, phys, mid, th = 1.0, [], [], None, None, 0.5, math.tanh
    loads = fem.cases if o.separate_load_cases else [sum(fem.cases)]
    for _ in range(o.max_iterations):
        soft = phys = flt.apply(rho)
        if o.enable_heaviside:  # beta stays 1 for the first 25 iterations
            phys = ((th(mid) + torch.tanh(soft - mid)) / (2 * th(mid))).clamp(0, 1)
        e = fem.young(phys)
        us = [fem.solve(e, f) for f in loads]
        comp.append(sum(float(f @ v) for f, v in zip(loads, us)))
        vol.append(float(phys.mean()))
        dc = -sum(o.penal * phys ** (o.penal - 1) * (fem.e0 - fem.emin) * fem.energy(v) for v in us)
        if o.enable_heaviside:
            dc = dc * (1 - torch.tanh(soft - mid) ** 2) / (2 * th(mid))
        rho, lam = _oc(rho, flt.adjoint(dc), flt.s, passive, o.volume_fraction, lam)
        u = sum(us)
    return dict(u=u.cpu().numpy(), physical=fem.box(phys).cpu().numpy().reshape(-1),
                design=fem.box(rho).cpu().numpy().reshape(-1), compliance=np.array(comp), volume=np.array(vol))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("many", "mesh"):  # trajectories of many solves; vertices chosen by FP32 comparisons
        return None
    ne = case["nx"] * case["ny"] * case["nz"]
    if kind == "update":
        st = prepare(case, seed)
        fem = _Fem(st["problem"].model)
        flt = _Cone(fem, case["rmin"])
        rho, u = fem.t(st["rho"]), fem.t(st["u"])
        phys = flt.apply(rho)
        ku = fem.apply(fem.young(phys), u)
        dc = flt.adjoint(-3.0 * phys ** 2 * (fem.e0 - fem.emin) * fem.energy(u))
        new, lam = _oc(rho, dc, flt.s, torch.zeros_like(rho, dtype=torch.bool), case["volfrac"], 1.0)
        return {k: (v.cpu().numpy() if isinstance(v, torch.Tensor) else v)
                for k, v in dict(physical=phys, ku=ku, dc=dc, rho=new, lam=lam).items()}
    solves = case.get("iterations", 1) * (case["loads"] if case.get("apart") else 1)
    if solves * (ne + 15_000) * max(case["nx"], case["ny"], case["nz"]) > 3e7:  # over about 20 seconds of Jacobi-PCG
        return None
    st = prepare(case, seed)
    if kind == "simp":
        return _exact_simp(st["model"], st["options"])
    fem = _Fem(st["model"])
    e = fem.young(fem.t(st["model"].element_density)[fem.active])
    f = sum(fem.cases)
    u = fem.solve(e, f)
    ku, react = fem.apply(e, u), torch.zeros_like(u)
    react[fem.fixed] = ku[fem.fixed]
    return dict(u=u.cpu().numpy(), compliance=float(f @ u),
                max_displacement=float(u.reshape(-1, 3).norm(dim=1).max()), reactions=react.cpu().numpy(),
                von_mises=fem.von_mises(e, u).cpu().numpy())
