"""Performance cases of the multiresolution advection path, through the package's public calls.

A case is one piece of work that a program built on this package does again and again: a time step of a large
adapted simulation, a run of some steps from a saved state, one evaluation of a right-hand side on arrays that
the program owns, a gradient by the adjoint, a step of an ensemble.  Meshes are 2D and 3D, from a few hundred
cells to millions; both stencil radii, both prediction radii, the upwind operator, the README lambda and the
flux form, periodic axes, vector fields, relative details and the batched mode occur, as the tests, the demos'
configurations and the benchmark use them.

prepare() makes what a program holds before the call: an adapted mesh with its fields (initial shapes drawn
from the seed, some steps run, so that no case starts on an unsmoothed jump), or the saved cells and values it
starts from.  run() is one pass; it returns the fields in samurai's reference numbering, in device buffers of a
size that the case alone decides (the first `reference` entries are the field), and the sizes of the mesh.
Runs ("run") begin at the same saved state in every pass.  Single steps ("step", "batch": large or many meshes,
which change little over the steps of a measurement) move the state on; the flow turns round every TURN steps,
so that the shapes stay in the box however many are made.
"""
import math
import random

import numpy as np
import torch

import samurai_gb300 as sg

TURN = 64  # steps after which the velocity of a stepping case changes sign


# ------------------------------------------------------------------ the cases
def _case(name, kind, **kw):
    c = dict(name=name, kind=kind, dim=2, min_level=2, max_level=8, radius=1, prediction=1, shapes=8, eps=1e-4, regularity=2.0,
             cfl=0.5, ax=1.0, ay=0.5, az=0.25, scheme=0, bc=0.0)
    c.update(kw)
    return c


def listed():
    return [
        # a member of a parameter sweep taken up from its saved state on a small mesh: latency and launches count
        _case("restart_2d_L6", "run", max_level=6, shapes=2, steps=1),
        # the README's program: levels 2 to 8, a square (and a Gaussian), velocity (1, 1)
        _case("readme_2d_L8", "run", max_level=8, shapes=2, ay=1.0, steps=10),
        # the advection demo's configuration: levels 4 to 10, epsilon 2e-4, regularity 1
        _case("demo_2d_L10", "run", min_level=4, max_level=10, shapes=3, eps=2e-4, regularity=1.0, ay=1.0, steps=12),
        # the benchmark's 2D workload: levels 4 to 12, 32 shapes
        _case("bench_2d_L12", "step", min_level=4, max_level=12, shapes=32),
        # a program with the library's default ghost width (2) and an odd level range
        _case("default_2d_L11", "run", min_level=3, max_level=11, radius=2, shapes=9, eps=1e-3, regularity=1.0, ay=-0.7, steps=12),
        # a flow on a doubly periodic box
        _case("periodic_2d_L9", "run", min_level=3, max_level=9, shapes=6, eps=1e-3, regularity=1.0, ax=0.8, ay=0.3, periodic=3, steps=10),
        # a system of three components adapted together on relative details
        _case("vector_2d_L9", "run", min_level=3, max_level=9, shapes=4, components=3, eps=1e-3, regularity=1.0, relative=True, steps=8),
        # 3D: an ordinary size and the benchmark's, the largest case
        _case("ball_3d_L7", "run", dim=3, min_level=2, max_level=7, shapes=5, eps=1e-3, regularity=1.0, cfl=0.3, ay=1.0, az=1.0, steps=8),
        # (its time step is short, as that of a program coupled to a faster process: the mesh stays alike over many steps)
        _case("ball_3d_L9", "step", dim=3, min_level=3, max_level=9, shapes=9, eps=1e-3, regularity=1.0, cfl=0.03, ay=1.0, az=1.0),
        # a program that integrates in time by itself: values in, ghosts and flux form, values out, on a uniform mesh
        _case("rhs_uniform_2d_L11", "rhs", min_level=11, max_level=11, scheme=2, bc=0.25, ax=0.9, ay=-0.4),
        # a gradient: sixteen steps recorded, then the reverse sweep
        _case("adjoint_2d_L9", "adjoint", min_level=3, max_level=9, shapes=6, ay=0.7, steps=16, checkpoint=8),
        # an ensemble stepped together: max_level 7 to 10, one to eight shapes each
        _case("batch_2d_48", "batch", instances=48, low=7, max_level=10, shapes=8, eps=1e-3, cfl=0.5),
    ]


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "rhs", "rhs", "adjoint", "batch"])
    dim = 3 if kind in ("run", "rhs") and rng.random() < 0.35 else 2
    sign = lambda: rng.choice([-1.0, 1.0])  # noqa: E731
    c = dict(kind=kind, dim=dim, radius=1, prediction=1, shapes=rng.randint(1, 12), eps=10 ** rng.uniform(-4, -2), regularity=rng.choice([0.0, 1.0, 2.0]),
             cfl=rng.uniform(0.1, 0.5) if dim == 2 else rng.uniform(0.1, 0.33), ax=sign() * rng.uniform(0.2, 1.0), ay=sign() * rng.uniform(0.2, 1.0),
             az=sign() * rng.uniform(0.2, 1.0), scheme=0, bc=rng.choice([0.0, rng.uniform(-1.0, 1.0)]))
    if dim == 2:
        c["max_level"] = rng.randint(5, 12) if kind == "run" else rng.randint(5, 10)
        c["min_level"] = rng.randint(2, min(5, c["max_level"] - 1))
    else:
        c["max_level"] = rng.randint(4, 8)
        c["min_level"] = rng.randint(2, 3)
    if kind == "rhs":
        if rng.random() < 0.5:
            c["min_level"] = c["max_level"] = rng.randint(4, 11) if dim == 2 else rng.randint(3, 7)
        c["scheme"] = rng.choice([0, 1, 2]) if dim == 2 else rng.choice([0, 2])
        if c["scheme"] == 1:  # the README's lambda is the velocity (1, 1)
            c["ax"], c["ay"] = 1.0, 1.0
    if kind == "run":
        c["steps"] = rng.randint(1, 12)
        c["scheme"] = rng.choice([0, 0, 2])
        if c["scheme"] != 2 and rng.random() < 0.25:
            c["periodic"] = rng.randint(1, (1 << dim) - 1)
        c["refine_boundary"] = rng.random() < 0.1
        c["radius"] = rng.choice([1, 1, 2])
        c["prediction"] = rng.choice([1, 1, 1, 0])
        if c["scheme"] == 0 and rng.random() < 0.25:
            c["components"] = rng.randint(2, 4)
            c["relative"] = rng.random() < 0.5
            c["max_level"] = min(c["max_level"], 10 if dim == 2 else 6)
            c["min_level"] = min(c["min_level"], c["max_level"] - 1)
    if kind == "adjoint":
        c["max_level"] = rng.randint(5, 9)
        c["min_level"] = rng.randint(2, 3)
        c["steps"] = rng.randint(3, 20)
        c["checkpoint"] = rng.randint(2, 9)
    if kind == "batch":
        c["instances"] = rng.randint(2, 48)
        c["low"] = rng.randint(6, 8)
        c["max_level"] = rng.randint(c["low"], 10)
    return c


# ------------------------------------------------------- initial shapes (torch, on the GPU)
def _shapes(rng, dim, n):
    """n bumps: boxes (2D) or balls (3D) and Gaussians in turn, sizes as the benchmark's"""
    out = []
    for k in range(n):
        centre = [rng.uniform(0.25, 0.75) for _ in range(dim)]
        amp = rng.uniform(0.5, 1.0)
        if k % 2 == 0:
            # half width or radius: with many shapes each is small, with few the size of the demos' disc
            size = rng.uniform(0.01, 0.05) if n > 12 else rng.uniform(0.08, 0.16)
            out.append(("box" if dim == 2 else "ball", size, centre, amp))
        else:
            out.append(("gauss", rng.uniform(0.005, 0.03) if dim == 2 else rng.uniform(0.01, 0.05), centre, amp))
    return out


def _values(shapes, level, coords):
    """the sum of the shapes at the cell centres (level: int tensor, coords: (n, dim) int tensor)"""
    length = torch.pow(2.0, -level.double())
    x = [length * (coords[:, d].double() + 0.5) for d in range(coords.shape[1])]
    u = torch.zeros_like(length)
    for kind, size, centre, amp in shapes:
        if kind == "box":
            inside = torch.ones_like(u, dtype=torch.bool)
            for d, c in enumerate(centre):
                inside &= (x[d] - c).abs() <= size
            u += amp * inside.double()
        else:
            r2 = sum((x[d] - c) ** 2 for d, c in enumerate(centre))
            u += amp * ((r2 <= size * size).double() if kind == "ball" else torch.exp(-r2 / (2.0 * size * size)))
    return u


def _uniform(mesh, dim, level):
    idx = np.arange(1 << level, dtype=np.int32)
    grids = np.meshgrid(*([idx] * dim), indexing="ij")
    coords = np.stack([g.ravel() for g in reversed(grids)], axis=1)
    mesh.set_cells(np.full(coords.shape[0], level, np.int32), coords)


def _upload(field, mesh, values_of):
    """field := values_of(level, coords) on the leaf cells, zero on the other reference cells"""
    level, coords, index = mesh.cells()
    dev = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    full = torch.zeros(mesh.nb_cells("reference"), dtype=torch.float64, device="cuda")
    full[dev(index)] = values_of(dev(level), dev(coords))
    torch.cuda.synchronize()
    field.upload_device(full.data_ptr(), full.numel())
    mesh.synchronize()
    return full


def _velocity(case):
    return [case["ax"], case["ay"], case["az"]][: case["dim"]]


def _dt(case):
    return case["cfl"] / (1 << case["max_level"])


def _room(case):
    """entries of a buffer that holds a field of any mesh of the case: never more than about 1.5 times the finest grid"""
    n, dim = 1 << case["max_level"], case["dim"]
    full = int(1.6 * (n + 6) ** dim) + 1024
    return full if case["min_level"] == case["max_level"] else min(full, int((400 if dim == 2 else 60) * n ** (dim - 1) * math.sqrt(case["shapes"])) + 1024)


class _Reader:
    """a field in samurai's numbering in a device buffer that the program keeps"""

    def __init__(self, case):
        self.buf = torch.zeros(_room(case), dtype=torch.float64, device="cuda")

    def __call__(self, field, n):
        if n > self.buf.numel():
            raise RuntimeError("the mesh has %d reference cells, the buffer room for %d" % (n, self.buf.numel()))
        field.download_device(self.buf.data_ptr(), n)
        return self.buf


class _Sim:
    """one adapted problem with the calls of the demos' time loop"""

    def __init__(self, case, seed, warm=24, shapes=None):
        self.case = case
        rng = random.Random(seed * 7919 + 17)
        dim, low, high = case["dim"], case["min_level"], case["max_level"]
        periodic = [bool(case.get("periodic", 0) >> d & 1) for d in range(dim)]
        n = case.get("components", 1)
        if n == 1:
            self.sim = sg.AdvectionSim(dim, low, high, case["radius"], case["prediction"], 1, case["bc"], periodic=periodic)
            self.mesh, self.u, self.unp1, self.adaptation = self.sim.mesh, self.sim.u, self.sim.unp1, self.sim.adaptation
        else:
            self.mesh = sg.MRMesh(dim, low, high, case["radius"], case["prediction"], 1, periodic=periodic)
            self.u = sg.make_vector_field("u", self.mesh, n)
            self.unp1 = sg.make_vector_field("unp1", self.mesh, n)
            sg.make_bc(sg.Dirichlet(1), self.u, *[case["bc"]] * n)
            self.adaptation = sg.make_MRAdapt(self.u)
        self.mesh.set_refine_boundary(bool(case.get("refine_boundary")))
        self.cfg = sg.mra_config().epsilon(case["eps"]).regularity(case["regularity"]).relative_detail(bool(case.get("relative")))
        self.a, self.dt, self.steps, self.passes = _velocity(case), _dt(case), 0, 0
        self.readers = [_Reader(case) for _ in range(n)]
        # a uniform mesh of a moderate level, refined where the shapes want it: adapt, take the shapes' values on
        # the new cells, adapt again
        drawn = [_shapes(rng, dim, shapes or case["shapes"]) for _ in range(n)]
        start = max(low, min(high - 1, 9 if dim == 2 else 6)) if high > low else high
        if start < high:
            _uniform(self.mesh, dim, start)
        for _ in range(high - start + 2 if high > low else 1):
            for f, s in zip(self.u.components(), drawn):
                _upload(f, self.mesh, lambda lv, co, s=s: _values(s, lv, co))
            if high > low:
                self.adaptation(self.cfg)
        for _ in range(warm if high > low else 0):
            self.step()
        self.steps = 0

    def zero(self):
        for f in self.unp1.components():
            f.fill(0.0)

    def step(self):
        a = self.a if self.steps // TURN % 2 == 0 else [-v for v in self.a]
        self.steps += 1
        self.passes = self.adaptation(self.cfg)
        self.zero()
        sg.update_ghost_mr(self.u)
        self.unp1.assign_upwind(self.u, a, self.dt, self.case["scheme"])
        sg.swap(self.u, self.unp1)

    def read(self):
        cells, ref = self.mesh.counts()
        out = [r(f, ref) for r, f in zip(self.readers, self.u.components())]
        return {"u": out, "cells": cells, "reference": ref, "passes": self.passes}


# ------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return {"kind": kind, "sim": _Sim(case, seed)}
    if kind == "run":
        # a saved state: the leaf cells and the values after a step, before the next one's adaptation
        sim = _Sim(case, seed)
        level, coords, _ = sim.mesh.cells()
        got = sim.read()
        sim.mesh.synchronize()
        return {"kind": kind, "sim": sim, "level": level, "coords": coords, "values": [v[: got["reference"]].clone() for v in got["u"]]}
    if kind == "rhs":
        # the program's own array of values on a fixed mesh
        sim = _Sim(case, seed)
        sim.zero()
        _, ref = sim.mesh.counts()
        g = torch.Generator(device="cuda").manual_seed(seed)
        if case["min_level"] == case["max_level"]:
            values = torch.rand(ref, generator=g, dtype=torch.float64, device="cuda")
        else:
            got = sim.read()
            sim.mesh.synchronize()
            values = got["u"][0][:ref].clone()
        return {"kind": kind, "sim": sim, "values": values, "out": _Reader(case)}
    if kind == "adjoint":
        sim = _Sim(case, seed, warm=2)
        room = _room(case)
        return {"kind": kind, "sim": sim, "adjoint": sg.Adjoint(sim.u, case["checkpoint"]), "u0": torch.from_numpy(sim.u.cell_values()).cuda(),
                "u_end": torch.zeros(room, dtype=torch.float64, device="cuda"), "g0": torch.zeros(room, dtype=torch.float64, device="cuda")}
    # a batch of problems of different sizes, velocities and shapes; the spread of sizes is the same for every seed
    rng = random.Random(seed * 104729 + 5)
    sims, dts, vel = [], [], []
    n, levels = case["instances"], case["max_level"] - case["low"] + 1
    for k in range(n):
        one = dict(case, max_level=case["low"] + k % levels, ax=rng.uniform(-1.0, 1.0), ay=rng.uniform(-1.0, 1.0))
        sims.append(_Sim(one, seed * 1000 + k, warm=2, shapes=1 + rng.randrange(case["shapes"])))
        dts.append(_dt(one))
        vel.append(_velocity(one))
    return {"kind": kind, "sims": sims, "batch": sg.Batch([s.sim for s in sims]), "dt": dts, "a": vel, "steps": 0}


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["sim"].step()
        return state["sim"].read()
    if kind == "run":
        s = state["sim"]
        s.mesh.set_cells(state["level"], state["coords"])
        for f, v in zip(s.u.components(), state["values"]):
            f.upload_device(v.data_ptr(), v.numel())
        for _ in range(s.case["steps"]):
            s.step()
        s.steps = 0
        return s.read()
    if kind == "rhs":
        s = state["sim"]
        s.u.upload_device(state["values"].data_ptr(), state["values"].numel())
        sg.update_ghost_mr(s.u)
        s.unp1.assign_upwind(s.u, s.a, s.dt, s.case["scheme"])
        return state["out"](s.unp1, state["values"].numel())
    if kind == "adjoint":
        # J = 0.5 |u_end|^2: the gradient that comes in is u_end itself
        s, adj = state["sim"], state["adjoint"]
        n = adj.record_ptr(state["u0"].data_ptr(), s.case["steps"], s.case["eps"], s.case["regularity"], s.a, s.dt)
        adj.final_ptr(state["u_end"].data_ptr(), n)
        ga = adj.backward_ptr(state["u_end"].data_ptr(), state["g0"].data_ptr())
        return {"u": state["u_end"], "g0": state["g0"], "ga": ga, "cells": n}
    a = state["a"] if state["steps"] // TURN % 2 == 0 else [[-v for v in r] for r in state["a"]]
    state["steps"] += 1
    c = state["sims"][0].case
    passes = state["batch"].step(c["eps"], c["regularity"], a, state["dt"], c["scheme"])
    state["batch"].update_ghost()  # the fields are read with their ghosts
    out, sizes = [], []
    for s in state["sims"]:
        cells, ref = s.mesh.counts()
        sizes.append((cells, ref))
        out.append(s.readers[0](s.u, ref))
    return {"u": out, "sizes": np.array(sizes, np.int64), "passes": np.array(passes, np.int32)}


# --------------------------------------------------------------------------- work
def _leaves(case):
    """about how many leaf cells the adapted mesh has: bands along the shapes' edges at the finest levels"""
    n = 1 << case["max_level"]
    if case["min_level"] == case["max_level"]:
        return n ** case["dim"]
    tight = (1e-3 / case["eps"]) ** 0.15
    if case["dim"] == 2:
        return min(n * n, 60 + 9.0 * tight * n * case["shapes"] ** 0.75)
    return min(n ** 3, 200 + 3.5 * tight * n * n * case["shapes"] ** 0.5)


def work(case):
    """One pass: the leaf values read and written (and, where the program's own array goes in or out, that array), the
    additions and products of the scheme: fluxes of the upwind step per leaf, 2 * 3^dim - 1 per child for the detail."""
    kind, dim = case["kind"], case["dim"]
    if kind == "batch":
        levels = case["max_level"] - case["low"] + 1
        n = sum(_leaves(dict(case, max_level=case["low"] + k % levels, shapes=1 + case["shapes"] / 2)) for k in range(case["instances"]))
    else:
        n = _leaves(case)
    n *= case.get("components", 1)
    upwind = 10 * dim + 2
    if kind == "rhs":
        return {"bytes": 16.0 * n, "flops": float(upwind * n)}
    step = upwind + 3 ** dim + 4
    if kind == "adjoint":
        return {"bytes": 32.0 * n * case["steps"], "flops": 3.0 * step * n * case["steps"]}
    return {"bytes": 16.0 * n * case.get("steps", 1), "flops": float(step * n * case.get("steps", 1))}


# -------------------------------------------------------------------------- exact
def exact(case, seed):
    """The right-hand side on a uniform mesh is a plain stencil (the flux form and the operator form agree there);
    adapted meshes have no closed form."""
    if case["kind"] != "rhs" or case["min_level"] != case["max_level"]:
        return None
    dim, n = case["dim"], 1 << case["max_level"]
    # the reference cells of a uniform mesh: the box and one layer around it, rows in order
    g = torch.Generator(device="cuda").manual_seed(seed)
    values = torch.rand((n + 2) ** dim, generator=g, dtype=torch.float64, device="cuda").reshape((n + 2,) * dim)
    inner = (slice(1, n + 1),) * dim
    u = values.clone()
    for d in range(dim):
        ax = dim - 1 - d
        for ghost, cell in ((0, 1), (n + 1, n)):
            u.select(ax, ghost).copy_(2.0 * case["bc"] - u.select(ax, cell))
    acc = torch.zeros((n,) * dim, dtype=torch.float64, device="cuda")
    for d, a in enumerate(_velocity(case)):
        ax = dim - 1 - d
        at = lambda o: u[tuple(slice(1 + (o if k == ax else 0), n + 1 + (o if k == ax else 0)) for k in range(dim))]  # noqa: E731,B023
        flux = lambda left, right: 0.5 * a * (left + right) + 0.5 * abs(a) * (left - right)  # noqa: E731,B023
        acc += flux(at(0), at(1)) - flux(at(-1), at(0))
    out = torch.zeros(_room(case), dtype=torch.float64, device="cuda")
    out[: u.numel()].view(u.shape)[inner] = u[inner] - case["cfl"] / n * math.ldexp(1.0, case["max_level"]) * acc
    return out
