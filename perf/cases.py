"""What this library is timed on: its public calls over the sizes they are used at.

Each case is one call, or the few calls a driver makes together, on a problem whose points,
materials and boundary conditions are in hand (``prepare``).  The sizes are those of the
library's own workloads (``gale_b200/workloads.py``); ``draw`` spreads the same kinds over
smaller, ragged and anisotropic meshes.  ``exact`` restates a case in plain FP64 torch where
that is possible.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from gale_b200 import abi, timeloop, workloads
from gale_b200.stokes import (BodyForce, DruckerPrager, FrankKamenetskii, MaterialViscosity, Mesh, Picard,
                              RheologyMaterial, StokesProblem, StrainWeakening, UzawaSolver, VelocityBC,
                              free_slip)

THETA, RAYLEIGH = 9.21, 1e6
PCDVC = dict(upperT=25.0, lowerT=0.6, maxSplits=3, maxDeletions=3)
BATCH_SIZES = (32, 48, 64, 96, 128)


def listed():
    return [
        # a step's remap of a host-owned swarm: elements of the creep model's 7.1 M points
        {"name": "locate_creep", "kind": "locate", "nx": 64, "ny": 64, "nz": 64, "ppc": 27},
        # the same search on a caller's own device buffers, at that entry point's largest mesh
        {"name": "locate_device_subduction", "kind": "locate_device", "nx": 128, "ny": 64, "nz": 128, "ppc": 27},
        # assembly of one Picard iteration of the extension model, yielding from a previous solution
        {"name": "assemble_extension", "kind": "assemble", "model": "extension", "nx": 256, "ny": 64, "nz": 0,
         "ppc": 40, "precision": "mixed"},
        # assembly of the creep model as a host shim reads it back
        {"name": "assemble_creep", "kind": "assemble", "model": "creep", "nx": 64, "ny": 64, "nz": 64, "ppc": 27,
         "precision": "mixed"},
        # Courant step and RK2 advection of the creep model's points
        {"name": "advect_creep", "kind": "advect", "nx": 64, "ny": 64, "nz": 64, "ppc": 27, "order": 2},
        # remap with Voronoi integration weights in 3D
        {"name": "weights_3d", "kind": "weights", "nx": 32, "ny": 32, "nz": 32, "ppc": 27, "res": 10},
        # remap, weights and population control of a host-owned 2D swarm
        {"name": "population_extension", "kind": "population", "nx": 256, "ny": 64, "nz": 0, "ppc": 40, "res": 10},
        # one whole PIC time step of the lid-driven regression model: the smallest problem
        {"name": "step_lid", "kind": "step", "nx": 20, "ny": 20, "ppc": 36, "res": 10},
        # the plain FP64 Uzawa solve, the default configuration, on the 2D sinker
        {"name": "solve_sinker_fp64", "kind": "solve", "model": "sinker", "nx": 64, "ny": 64, "nz": 0, "ppc": 20,
         "precision": "fp64", "inner": "jacobi", "tolerance": 1e-5, "degree": 0},
        # operator build and mixed multigrid solve of the 3D creep model
        {"name": "solve_creep_mixed", "kind": "solve", "model": "creep", "nx": 64, "ny": 64, "nz": 64, "ppc": 27,
         "precision": "mixed", "inner": "mg", "tolerance": 1e-6, "degree": 3},
        # the non-linear extension model, 20 Picard iterations
        {"name": "picard_extension", "kind": "picard", "nx": 256, "ny": 64, "ppc": 40, "iterations": 20},
        # an uneven batch of independent 2D problems
        {"name": "batch_sinkers", "kind": "batch", "count": 128, "ppc": 20, "max_size": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("locate", "locate_device", "assemble", "advect", "advect", "weights", "population", "step",
                       "solve", "solve", "picard", "batch"))
    flat = rng.random() < 0.5
    if kind in ("locate", "locate_device", "advect"):
        n = ({"nx": _log(rng, 8, 400), "ny": _log(rng, 8, 400), "nz": 0} if flat else
             {"nx": _log(rng, 4, 64), "ny": _log(rng, 4, 64), "nz": _log(rng, 4, 64)})
        c = {"kind": kind, **n, "ppc": rng.randint(8, 27)}
        return dict(c, order=rng.choice((1, 2))) if kind == "advect" else c
    if kind == "assemble":
        prec = rng.choice(("fp64", "mixed"))
        if flat:
            return {"kind": kind, "model": "extension", "nx": _log(rng, 16, 256), "ny": _log(rng, 8, 64), "nz": 0,
                    "ppc": rng.randint(16, 40), "precision": prec}
        return {"kind": kind, "model": "creep", "nx": _log(rng, 4, 64), "ny": _log(rng, 4, 64),
                "nz": _log(rng, 4, 64), "ppc": rng.randint(8, 27), "precision": prec}
    if kind in ("weights", "population"):
        if flat:
            return {"kind": kind, "nx": _log(rng, 8, 256), "ny": _log(rng, 8, 64), "nz": 0,
                    "ppc": rng.randint(16, 40), "res": rng.choice((7, 10, 15))}
        return {"kind": kind, "nx": _log(rng, 4, 32), "ny": _log(rng, 4, 32), "nz": _log(rng, 4, 32),
                "ppc": rng.randint(16, 27), "res": rng.choice((7, 10))}
    if kind == "step":
        return {"kind": kind, "nx": rng.randint(12, 28), "ny": rng.randint(12, 28), "ppc": rng.randint(20, 36),
                "res": 10}
    if kind == "solve":
        if flat:
            return {"kind": kind, "model": "sinker", "nx": _log(rng, 16, 72), "ny": _log(rng, 16, 72), "nz": 0,
                    "ppc": rng.randint(12, 24), "precision": "fp64", "inner": "jacobi", "tolerance": 1e-5,
                    "degree": 0}
        nx, ny, nz = (8 * rng.randint(2, 8) for _ in range(3))
        return {"kind": kind, "model": "creep", "nx": nx, "ny": ny, "nz": nz, "ppc": rng.randint(12, 27),
                "precision": "mixed", "inner": "mg", "tolerance": rng.choice((1e-5, 1e-6)),
                "degree": rng.choice((0, 3))}
    if kind == "picard":
        return {"kind": kind, "nx": 32 * rng.randint(2, 8), "ny": 16 * rng.randint(1, 4), "ppc": rng.randint(24, 40),
                "iterations": rng.randint(3, 20)}
    return {"kind": kind, "count": 2 * _log(rng, 2, 64), "ppc": rng.randint(12, 20), "max_size": rng.choice((64, 96, 128))}


# ------------------------------------------------------------------------ inputs ----
def _extent(case):
    """Domain of a case: square 2D elements on [0, nx/ny] × [0, 1] for the extension model and
    the swarms of that shape, the unit box otherwise."""
    if case.get("model") == "extension" or case["kind"] in ("population", "picard"):
        if not case.get("nz"):
            return (case["nx"] / case["ny"], 1.0)
    return (1.0, 1.0, 1.0) if case.get("nz") else (1.0, 1.0)


def _mesh(case):
    n = [case["nx"], case["ny"]] + ([case["nz"]] if case.get("nz") else [])
    return Mesh(len(n), n, (0.0,) * len(n), _extent(case))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _points(mesh, ppc, gen):
    """ppc uniform-random points in every element, shuffled: [np, dim] on the GPU."""
    dim = mesh.dim
    nel = math.prod(mesh.elements[d] for d in range(dim))
    e = torch.arange(nel, device="cuda").repeat_interleave(ppc)
    e = e[torch.randperm(nel * ppc, generator=gen, device="cuda")]
    x = torch.empty(nel * ppc, dim, dtype=torch.float64, device="cuda")
    for d in range(dim):
        n = mesh.elements[d]
        t = torch.rand(nel * ppc, generator=gen, dtype=torch.float64, device="cuda").clamp_(1e-6, 1 - 1e-6)
        x[:, d] = mesh.min[d] + (e % n + t) / n * (mesh.max[d] - mesh.min[d])
        e = e // n
    return x


def _nodes(mesh):
    return torch.as_tensor(workloads.node_coords(mesh), device="cuda")


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _roll(mesh, gen):
    """A nodal velocity that is tangential on every wall: convection rolls of random strength."""
    x = _nodes(mesh)
    a = torch.rand(4, generator=gen, dtype=torch.float64, device="cuda") + 0.5
    s = [(x[:, d] - mesh.min[d]) / (mesh.max[d] - mesh.min[d]) * math.pi for d in range(mesh.dim)]
    u = torch.zeros_like(x)
    u[:, 0] = a[0] * torch.sin(s[0]) * torch.cos(s[1]) + 0.3 * a[1] * torch.sin(2 * s[0]) * torch.cos(2 * s[1])
    u[:, 1] = -a[0] * torch.cos(s[0]) * torch.sin(s[1]) - 0.3 * a[1] * torch.cos(2 * s[0]) * torch.sin(2 * s[1])
    if mesh.dim == 3:
        u[:, 2] = 0.5 * a[2] * torch.sin(s[2]) * torch.cos(s[1])
    for d in range(mesh.dim):
        n = torch.arange(x.shape[0], device="cuda")
        for o in range(d):
            n = n // (mesh.elements[o] + 1)
        n = n % (mesh.elements[d] + 1)
        u[(n == 0) | (n == mesh.elements[d]), d] = 0.0
    return u


class _Inputs:
    """The arrays and tables of one problem, on the GPU where `exact` reads them."""

    def __init__(self, case, seed):
        kind, model = case["kind"], case.get("model")
        if kind == "picard" or kind == "population":
            model = "extension"
        gen = _generator(seed)
        self.mesh = m = _mesh(case)
        self.x = _points(m, case["ppc"], gen)
        self.T = self.plastic = self.prev = None
        y = self.x[:, 1]
        if model == "extension":
            self.material = torch.where(y >= 0.75, 2, torch.where(y >= 0.5, 1, 0)).int()
            r = torch.rand(y.shape[0], generator=gen, dtype=torch.float64, device="cuda")
            self.plastic = torch.where(self.material == 2, 0.1 * r, torch.zeros_like(r))
            sw = StrainWeakening(initialSofteningStrain=0.0, finalSofteningStrain=0.5)
            dp = DruckerPrager(cohesion=1.0, cohesionAfterSoftening=0.1, frictionCoefficient=0.6,
                               frictionCoefficientAfterSoftening=0.6, strainWeakening=True)
            self.mats = [RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
                         RheologyMaterial([MaterialViscosity(1e2)], density=1.0),
                         RheologyMaterial([MaterialViscosity(1e3), dp], density=1.0, strainWeakening=sw)]
            self.bc = VelocityBC(left={"vx": -1.0}, right={"vx": 1.0}, bottom={"vy": 0.0})
            self.force = BodyForce(gravity=1.0)
            if m.dim == 2:
                self.prev = self._stretching(m, gen)
        elif model == "sinker":
            c = torch.rand(3, generator=gen, dtype=torch.float64, device="cuda")
            r2 = (self.x[:, 0] - 0.4 - 0.2 * c[0]) ** 2 + (y - 0.7 - 0.1 * c[1]) ** 2
            self.material = (r2 < (0.08 + 0.04 * c[2]) ** 2).int()
            self.mats = [RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
                         RheologyMaterial([MaterialViscosity(100.0)], density=1.01)]
            self.bc, self.force = free_slip(m.dim), BodyForce(gravity=1.0)
        else:  # temperature-dependent creep; also the swarm of the remap and advection cases
            self.material = torch.zeros(y.shape[0], dtype=torch.int32, device="cuda")
            n = _nodes(m)
            self.T = 1.0 - n[:, 1] + 0.05 * torch.randn(n.shape[0], generator=gen, dtype=torch.float64,
                                                       device="cuda")
            self.mats = [RheologyMaterial([FrankKamenetskii(eta0=math.exp(0.5 * THETA), theta=THETA)])]
            self.bc, self.force = free_slip(m.dim), BodyForce(rayleighNumber=RAYLEIGH)
        self.u = _roll(m, gen)

    def _stretching(self, m, gen):
        """A stretching flow with a few shear zones, and a lithostatic pressure."""
        n = _nodes(m)
        w = m.max[0]
        a = torch.rand(3, generator=gen, dtype=torch.float64, device="cuda")
        u = torch.stack([2.0 * n[:, 0] / w - 1.0, -2.0 * n[:, 1] / w], 1)
        u[:, 0] += 0.1 * a[0] * torch.sin(7.0 * n[:, 0]) * torch.sin(math.pi * n[:, 1])
        u[:, 1] += 0.1 * a[1] * torch.cos(5.0 * n[:, 0]) * n[:, 1]
        ey = (torch.arange(m.elements[1], device="cuda", dtype=torch.float64) + 0.5) / m.elements[1]
        p = (1.0 - ey).repeat_interleave(m.elements[0]) * (1.0 + 0.1 * a[2])
        return u, p

    def problem(self):
        self.hx, self.hm = _host(self.x), _host(self.material)
        self.hp = None if self.plastic is None else _host(self.plastic)
        prob = StokesProblem(self.mesh)
        prob.set_velocity_bc(self.bc)
        prob.set_materials(self.mats)
        prob.set_body_force(self.force)
        if self.T is not None:
            prob.set_temperature(_host(self.T))
        prob.set_points(self.hx, self.hm, self.hp)
        return prob


def _lid(case, seed):
    """The lid-driven PIC model: no-flow walls, a partial lid on top, one fluid."""
    mesh = _mesh(case)
    gen = _generator(seed)
    nodes = workloads.node_coords(mesh)
    nx, ny = mesh.elements[0] + 1, mesh.elements[1]
    ix, iy = np.arange(nodes.shape[0]) % nx, np.arange(nodes.shape[0]) // nx
    fixed = np.zeros(nodes.shape[0], dtype=np.uint8)
    values = np.zeros((nodes.shape[0], 2))
    fixed[iy == 0] |= 2
    fixed[(ix == 0) | (ix == nx - 1)] |= 1
    fixed[iy == ny] |= 3
    values[iy == ny, 0] = workloads.partial_lid_top_layer(mesh, nodes[iy == ny, 0])
    x = _host(_points(mesh, case["ppc"], gen))
    prob = StokesProblem(mesh)
    prob.set_velocity_bc_nodes(fixed, values)
    prob.set_materials([RheologyMaterial([MaterialViscosity(1.0)])])
    prob.set_body_force(BodyForce())
    return {"prob": prob, "x": x, "m": np.zeros(x.shape[0], dtype=np.int32), "out": _swarm(mesh, 2 * x.shape[0]),
            "params": UzawaSolver(tolerance=1e-5, maxIterations=5000)}


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    gen = _generator(seed)
    sizes = [s for s in BATCH_SIZES if s <= case["max_size"]]
    probs = []
    for i in range(case["count"]):
        n = sizes[(7 * i) % len(sizes)]
        eta, r = 10 ** rng.uniform(0.0, 4.0), rng.uniform(0.05, 0.2)
        mesh = Mesh(2, (n, n), (0.0, 0.0), (1.0, 1.0))
        x = _points(mesh, case["ppc"], gen)
        m = ((x[:, 0] - 0.5) ** 2 + (x[:, 1] - 0.75) ** 2 < r * r).int()
        prob = StokesProblem(mesh)
        prob.set_velocity_bc(free_slip(2))
        prob.set_materials([RheologyMaterial([MaterialViscosity(1.0)], density=1.0),
                            RheologyMaterial([MaterialViscosity(eta)], density=1.01)])
        prob.set_body_force(BodyForce(gravity=1.0))
        prob.set_points(_host(x), _host(m))
        probs.append(prob)
    return {"probs": probs, "params": UzawaSolver(tolerance=1e-5, precision="mixed", inner="mg")}


def _swarm(mesh, np0):
    """A host's arrays for the points after population control, at their largest count."""
    n = np0 + PCDVC["maxSplits"] * math.prod(mesh.elements[d] for d in range(mesh.dim))
    return {"coords": np.zeros((n, mesh.dim)), "material": np.zeros(n, dtype=np.int32), "plastic": np.zeros(n),
            "xi": np.zeros((n, mesh.dim)), "w": np.zeros(n)}


def _read_points(prob, out):
    """The points and integration points through the C interface, into the host's arrays."""
    prob._check(prob.lib.gg_get_points(prob.h, abi.ptr(out["coords"]), abi.ptr(out["material"], C.c_int32),
                                       abi.ptr(out["plastic"])))
    prob._check(prob.lib.gg_get_integration_points(prob.h, abi.ptr(out["xi"]), abi.ptr(out["w"])))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return {"kind": kind, "res": case["res"], **_lid(case, seed)}
    if kind == "batch":
        return {"kind": kind, **_batch(case, seed)}
    if kind == "locate_device":
        mesh = _mesh(case)
        x = _points(mesh, case["ppc"], _generator(seed))
        nel = math.prod(mesh.elements[d] for d in range(mesh.dim))
        new = lambda n: torch.zeros(n, dtype=torch.int32, device="cuda")  # noqa: E731
        return {"kind": kind, "lib": abi.load_library(), "mesh": mesh, "x": x, "cell": new(x.shape[0]),
                "offsets": new(nel + 1), "order": new(x.shape[0])}
    inp = _Inputs(case, seed)
    s = {"kind": kind, "prob": inp.problem()}
    if kind == "locate":
        return s
    if kind == "advect":
        return dict(s, u=_host(inp.u), order=case["order"])
    if kind == "weights":
        s["prob"].set_weights("dvc", case["res"])
        return s
    if kind == "population":
        s["prob"].set_weights("dvc", case["res"])
        return dict(s, points=(inp.hx, inp.hm, inp.hp), out=_swarm(inp.mesh, inp.hx.shape[0]))
    s["prob"].locate()
    if kind == "assemble":
        prev = None if inp.prev is None else tuple(_host(v).reshape(-1) for v in inp.prev)
        return dict(s, precision=case["precision"], prev=prev)
    if kind == "picard":
        return dict(s, picard=Picard(nonLinearMaxIterations=case["iterations"], nonLinearTolerance=1e-5),
                    params=UzawaSolver(tolerance=1e-5, precision="mixed", inner="mg"))
    return dict(s, precision=case["precision"],
                params=UzawaSolver(tolerance=case["tolerance"], precision=case["precision"], inner=case["inner"],
                                   smoothingDegree=case["degree"]))


# --------------------------------------------------------------------------- run ----
def run(s):
    kind = s["kind"]
    if kind == "locate":
        return s["prob"].locate()
    if kind == "locate_device":
        outside, msg = C.c_int64(0), C.c_char_p()
        rc = s["lib"].gg_locate_noalloc(C.byref(s["mesh"]), s["x"].shape[0], s["x"].data_ptr(),
                                        s["cell"].data_ptr(), s["offsets"].data_ptr(), s["order"].data_ptr(),
                                        C.byref(outside), torch.cuda.current_stream().cuda_stream, C.byref(msg))
        if rc != 0:
            raise RuntimeError(msg.value.decode())
        return s["cell"], s["offsets"], s["order"]
    if kind == "assemble":
        prob = s["prob"]
        prob.build_operator(s["precision"], s["prev"])
        f, h = prob.rhs()
        kd, sd = prob.diagonals()
        return {"f": f, "h": h, "k_diag": kd, "schur_diag": sd}
    if kind == "advect":
        dt = s["prob"].courant_dt(s["u"])
        return {"dt": dt, "coords": s["prob"].advect(dt, s["u"], s["order"])}
    if kind == "weights":
        cell = s["prob"].locate()
        xi, w = s["prob"].integration_points()
        return {"cell": cell, "xi": xi, "w": w}
    if kind == "population":
        prob = s["prob"]
        prob.set_points(*s["points"])
        prob.locate()
        st = prob.population_control(**PCDVC)
        return {"splits": st["splits"], "deletions": st["deletions"], **_read_points(prob, s["out"])}
    if kind == "step":
        s["prob"].set_points(s["x"], s["m"])
        r = timeloop.run_pic_steps(s["prob"], s["params"], 1, PCDVC, s["res"])
        s["out"]["coords"][:r["coords"].shape[0]] = r["coords"]
        s["out"]["material"][:r["material"].shape[0]] = r["material"]
        return {"u": r["u"], "p": r["p"], "dt": r["dt"], "points": r["coords"].shape[0],
                "coords": s["out"]["coords"], "material": s["out"]["material"]}
    if kind == "solve":
        s["prob"].build_operator(s["precision"])
        u, p, _ = s["prob"].solve(s["params"])
        return {"u": u, "p": p}
    if kind == "picard":
        u, p, _ = s["prob"].picard(s["picard"], s["params"])
        return {"u": u, "p": p}
    r = StokesProblem.solve_batch(s["probs"], s["params"])
    return {"u": np.concatenate([x[0] for x in r]), "p": np.concatenate([x[1] for x in r])}


# -------------------------------------------------------------------------- work ----
def work(case):
    """Inputs read once and outputs written once; operations of the per-point evaluations."""
    kind, ppc = case["kind"], case["ppc"]
    if kind == "batch":
        sizes = [s for s in BATCH_SIZES if s <= case["max_size"]]
        nel = case["count"] * sum(n * n for n in sizes) / len(sizes)
        nn, dim = case["count"] * sum((n + 1) ** 2 for n in sizes) / len(sizes), 2
    else:
        n = [case["nx"], case["ny"]] + ([case["nz"]] if case.get("nz") else [])
        nel, nn, dim = math.prod(n), math.prod(k + 1 for k in n), len(n)
    pts, nen = nel * ppc, 2 ** dim
    solution = 8 * (dim * nn + nel)
    point = 8 * dim + 4
    if kind == "locate":
        return {"bytes": pts * (8 * dim + 4), "flops": pts * 4 * dim}
    if kind == "locate_device":
        return {"bytes": pts * (8 * dim + 8) + 4 * nel, "flops": pts * 4 * dim}
    if kind == "advect":
        return {"bytes": pts * 16 * dim + 8 * dim * nn, "flops": case["order"] * pts * nen * (2 * dim + dim)}
    if kind in ("weights", "population"):
        cells = nel * case["res"] ** dim
        return {"bytes": pts * (8 * dim + 8 * (dim + 1) + 4), "flops": cells * 5 * dim}
    moments = pts * 2 * (23 if dim == 3 else 6)
    if kind == "assemble":
        return {"bytes": pts * point + 16 * dim * nn + 16 * nel, "flops": moments}
    return {"bytes": pts * point + solution, "flops": moments}


# ------------------------------------------------------------------------- exact ----
def _cells(mesh, x):
    idx = [torch.floor((x[:, d] - mesh.min[d]) / ((mesh.max[d] - mesh.min[d]) / mesh.elements[d]))
           .long().clamp_(0, mesh.elements[d] - 1) for d in range(mesh.dim)]
    e, stride = torch.zeros_like(idx[0]), 1
    for d in range(mesh.dim):
        e += idx[d] * stride
        stride *= mesh.elements[d]
    return e, idx


class _Elements:
    """Corner nodes, shape functions and their gradients at points of a regular mesh."""

    def __init__(self, mesh, x):
        self.mesh, self.dim = mesh, mesh.dim
        self.h = [(mesh.max[d] - mesh.min[d]) / mesh.elements[d] for d in range(mesh.dim)]
        self.e, idx = _cells(mesh, x)
        self.xi = [2.0 * ((x[:, d] - mesh.min[d]) / self.h[d] - idx[d]) - 1.0 for d in range(mesh.dim)]
        self.idx = idx

    def node(self, a):
        n, stride = 0, 1
        for d in range(self.dim):
            n = n + (self.idx[d] + ((a >> d) & 1)) * stride
            stride *= self.mesh.elements[d] + 1
        return n

    def N(self, a):
        v = 1.0
        for d in range(self.dim):
            v = v * 0.5 * (1.0 + (self.xi[d] if (a >> d) & 1 else -self.xi[d]))
        return v

    def dN(self, a, d):
        v = (1.0 if (a >> d) & 1 else -1.0) / self.h[d]
        for o in range(self.dim):
            if o != d:
                v = v * 0.5 * (1.0 + (self.xi[o] if (a >> o) & 1 else -self.xi[o]))
        return v if torch.is_tensor(v) else torch.full_like(self.xi[0], v)


def _velocity(el, u):
    v = 0.0
    for a in range(2 ** el.dim):
        v = v + u[el.node(a)] * el.N(a)[:, None]
    return v


def _viscosity(case, inp, el):
    if inp.T is not None:
        T = sum(inp.T[el.node(a)] * el.N(a) for a in range(2 ** el.dim))
        return math.exp(0.5 * THETA) * torch.exp(-THETA * T), T
    if case["kind"] == "solve":
        return torch.where(inp.material == 1, 100.0, 1.0).double(), None
    u, p = inp.prev
    g = [[sum(u[el.node(a), c] * el.dN(a, d) for a in range(4)) for d in range(2)] for c in range(2)]
    xx, yy, xy = g[0][0], g[1][1], 0.5 * (g[0][1] + g[1][0])
    tr = 0.5 * (xx + yy)
    inv = torch.sqrt(0.5 * ((xx - tr) ** 2 + (yy - tr) ** 2) + xy ** 2)
    ratio = (inp.plastic / 0.5).clamp(0.0, 1.0)
    C = 1.0 * (1 - ratio) + 0.1 * ratio
    f = 1.0 / math.sqrt(1.0 + 0.6 * 0.6)
    crit = torch.maximum(0.6 * p[el.e] * f + C * f, C * f)
    eta = torch.where(inp.material == 2, 1e3, torch.where(inp.material == 1, 1e2, 1.0)).double()
    yields = (inp.material == 2) & (crit < 2.0 * eta * inv)
    return torch.where(yields, crit / (2.0 * inv), eta), None


def _boundary(mesh, bc):
    """Fixed mask and values [nodes, dim] of the wall conditions."""
    nn = math.prod(mesh.elements[d] + 1 for d in range(mesh.dim))
    mask = torch.zeros(nn, mesh.dim, dtype=torch.bool, device="cuda")
    val = torch.zeros(nn, mesh.dim, dtype=torch.float64, device="cuda")
    n = torch.arange(nn, device="cuda")
    for d in range(mesh.dim):
        i = n % (mesh.elements[d] + 1)
        n = n // (mesh.elements[d] + 1)
        for side, on in ((0, i == 0), (1, i == mesh.elements[d])):
            for c in range(mesh.dim):
                if bc.fixed[2 * d + side][c]:
                    mask[on, c] = True
                    val[on, c] = bc.value[2 * d + side][c]
    return mask, val


def _assembled(case, inp):
    """Force, divergence right-hand side, diagonals and the point data of the operator."""
    m = inp.mesh
    dim, nen = m.dim, 2 ** m.dim
    el = _Elements(m, inp.x)
    nel = math.prod(m.elements[d] for d in range(dim))
    nn = math.prod(m.elements[d] + 1 for d in range(dim))
    eta, T = _viscosity(case, inp, el)
    count = torch.bincount(el.e, minlength=nel).double()
    vol = math.prod(el.h)
    c = vol / count[el.e]
    mask, val = _boundary(m, inp.bc)
    f = torch.zeros(nn, dim, dtype=torch.float64, device="cuda")
    if T is not None:
        body = RAYLEIGH * T
    else:
        rho = (torch.where(inp.material == 1, 1.01, 1.0) if case["kind"] == "solve" else
               torch.ones(inp.x.shape[0], device="cuda")).double()
        body = -rho
    ke = torch.zeros(nen, dim, nel, dtype=torch.float64, device="cuda")
    fixed = val.abs().sum() > 0
    if fixed:
        g = [[sum(val[el.node(a), i] * el.dN(a, d) for a in range(nen)) for d in range(dim)] for i in range(dim)]
    for a in range(nen):
        n, N = el.node(a), el.N(a)
        f[:, 1].index_add_(0, n, c * body * N)
        d2 = [el.dN(a, d) ** 2 for d in range(dim)]
        for i in range(dim):
            ke[a, i].index_add_(0, el.e, c * eta * (sum(d2) + d2[i]))
            if fixed:
                t = sum((g[i][d] + g[d][i]) * el.dN(a, d) for d in range(dim))
                f[:, i].index_add_(0, n, -c * eta * t)
    f[mask] = 0.0
    # G_e: −∫ ∂N_a/∂x_c over the element
    e = torch.arange(nel, device="cuda")
    idx, r = [], e
    for d in range(dim):
        idx.append(r % m.elements[d])
        r = r // m.elements[d]
    kd = torch.zeros(nn, dim, dtype=torch.float64, device="cuda")
    sd = torch.zeros(nel, dtype=torch.float64, device="cuda")
    h = torch.zeros(nel, dtype=torch.float64, device="cuda")
    ge, nodes = [], []
    for a in range(nen):
        n, stride = 0, 1
        for d in range(dim):
            n = n + (idx[d] + ((a >> d) & 1)) * stride
            stride *= m.elements[d] + 1
        nodes.append(n)
        row = []
        for i in range(dim):
            G = -(1.0 if (a >> i) & 1 else -1.0) * vol / el.h[i] / 2 ** (dim - 1)
            row.append(G)
            kd[:, i].index_add_(0, n, ke[a, i])
            sd += G * G / ke[a, i]
            h -= G * val[n, i]
        ge.append(row)
    return {"f": f, "h": h, "kd": kd, "sd": sd, "el": el, "ceta": c * eta, "mask": mask, "val": val, "ge": ge,
            "nodes": nodes, "nel": nel, "nn": nn}


def _solution(case, inp):
    """Velocity of the discrete problem by a dense direct solve (pressure is free up to a constant)."""
    A = _assembled(case, inp)
    dim, el, nn, nel = inp.mesh.dim, A["el"], A["nn"], A["nel"]
    nd, nen = nn * dim, 2 ** dim
    M = torch.zeros(nd + nel, nd + nel, dtype=torch.float64, device="cuda")
    flat = M.view(-1)
    grad = [[el.dN(a, d) for d in range(dim)] for a in range(nen)]
    for a in range(nen):
        for b in range(nen):
            dot = sum(grad[a][d] * grad[b][d] for d in range(dim))
            for i in range(dim):
                for j in range(dim):
                    v = grad[a][j] * grad[b][i] + (dot if i == j else 0.0)
                    ke = torch.zeros(nel, dtype=torch.float64, device="cuda").index_add_(0, el.e, A["ceta"] * v)
                    rows, cols = A["nodes"][a] * dim + i, A["nodes"][b] * dim + j
                    flat.index_add_(0, rows * (nd + nel) + cols, ke)
    e = torch.arange(nel, device="cuda")
    for a in range(nen):
        for i in range(dim):
            rows = A["nodes"][a] * dim + i
            M[rows, nd + e] = A["ge"][a][i]
            M[nd + e, rows] = A["ge"][a][i]
    fixed = A["mask"].reshape(-1).nonzero()[:, 0]
    scale = A["kd"].mean()
    M[fixed, :] = 0.0
    M[:, fixed] = 0.0
    M[fixed, fixed] = scale
    M[nd:, nd:] -= 1.0 / (scale * nel)
    b = torch.cat([A["f"].reshape(-1), A["h"]])
    return torch.linalg.solve(M, b)[:nd] + A["val"].reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("locate", "locate_device"):
        mesh = _mesh(case)
        x = _points(mesh, case["ppc"], _generator(seed))
        cell, _ = _cells(mesh, x)
        if kind == "locate":
            return _host(cell.int()).astype(np.uint32)
        nel = math.prod(mesh.elements[d] for d in range(mesh.dim))
        offsets = torch.zeros(nel + 1, dtype=torch.int32, device="cuda")
        offsets[1:] = torch.bincount(cell, minlength=nel).cumsum(0)
        return cell.int(), offsets, torch.sort(cell, stable=True).indices.int()
    if kind == "assemble":
        A = _assembled(case, _Inputs(case, seed))
        return {"f": _host(A["f"].reshape(-1)), "h": _host(A["h"]), "k_diag": _host(A["kd"].reshape(-1)),
                "schur_diag": _host(A["sd"])}
    if kind == "advect":
        inp = _Inputs(case, seed)
        m = inp.mesh
        sep = min((m.max[d] - m.min[d]) / m.elements[d] for d in range(m.dim))
        dt = 0.5 * sep / float(inp.u.square().sum(1).max().sqrt())
        v = _velocity(_Elements(m, inp.x), inp.u)
        if case["order"] == 2:
            v = _velocity(_Elements(m, inp.x + 0.5 * dt * v), inp.u)
        return {"dt": dt, "coords": _host(inp.x + dt * v)}
    if kind == "solve":
        dim = 3 if case["nz"] else 2
        n = [case["nx"], case["ny"], case["nz"]][:dim]
        if dim * math.prod(k + 1 for k in n) + math.prod(n) > 20000:
            return None
        return {"u": _host(_solution(case, _Inputs(case, seed))), "p": None}
    return None
