"""The work that users of this package have it do, as timed cases.

``listed()`` names the cases and says what each stands for; ``draw(rng)`` gives
more of the same ranges.  ``prepare(case, seed)`` makes what a program has in
hand before the call, ``run(state)`` is one pass through the public entry
points, ``work(case)`` the bytes and operations it cannot do without and
``exact(case, seed)`` the same results in 64-bit torch.

A pass is a whole simulation from its initial state: ``MPMExplicit.solve_jit``,
the engine's restart (write the state, initialise, step, read), a recorded run
with its adjoint, or the same for a batch.  Restarting is what parameter
sweeps, inverse problems and data generation do, and it keeps every pass the
same.  Initial velocities are smooth seeded modes (a fraction of the wave
speed), particles sit at jittered Gauss points, as in the package's workloads.
"""
import math
import random

import numpy as np
import torch

import diffmpm_gb300 as D
from diffmpm_gb300.autograd import explicit_run

GRAVITY = (0.0, -9.81)
FLUSH = 1e-12
STATE = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid")
RESULT = ("loc", "velocity", "stress", "strain")


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _plane(name, kind, nx, ny, box, steps, **more):
    """A 2-D case: mesh nx x ny on [0, size] wide, particles in the cells of
    the fractions ``box`` = (x0, x1, y0, y1), side x side points a cell."""
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "x0": box[0], "x1": box[1], "y0": box[2],
         "y1": box[3], "steps": steps, "side": 2, "scheme": "usf", "material": "elastic", "E": 1e6,
         "nu": 0.25, "rho": 2000.0, "cfl": 0.1, "size": 1.0, "amp": 1e-3, "drift": 0.0,
         "reinit": True, "velocity_update": False, "checkpoint": 100}
    c.update(more)
    return c


def _bar(name, kind, nx, ppe, steps, **more):
    c = {"name": name, "kind": kind, "nx": nx, "ppe": ppe, "steps": steps, "scheme": "usf", "E": 1e6,
         "rho": 1000.0, "dt": 2e-4, "v0": 0.05, "gravity": -9.81, "force": 2.0}
    c.update(more)
    return c


def _batch(name, kind, members, spec, steps, **more):
    c = {"name": name, "kind": kind, "members": members, "spec": spec, "lo": 32, "hi": 256,
         "steps": steps, "checkpoint": 100}
    c.update(more)
    return c


def listed():
    return [
        # the smallest 2-D run, as in the package's smoke test: 144 particles,
        # 1000 steps in one call; launches and latency are all of it
        _plane("solve_small", "solve", 10, 10, (0.2, 0.8, 0.2, 0.8), 1000, E=1e4, nu=0.3, rho=1000.0, cfl=0.0037),
        # an ordinary deck: a block under a ramped traction on its top layer
        # and a ramped nodal force, on a mesh that is no multiple of anything
        _plane("solve_traction", "solve_loads", 118, 67, (0.1, 0.85, 0.0, 0.7), 250, nu=0.3, rho=1800.0),
        # 1-D: a bar under gravity and an end force, and the gradient of the
        # one-particle example (1000 USL steps) in its Young's modulus
        _bar("line_bar", "line", 60, 4, 500),
        _bar("line_grad", "line_grad", 1, 1, 1000, scheme="usl", E=100.0, rho=1.0, dt=0.01, v0=0.1,
             gravity=0.0, force=0.0),
        # material in motion: a soft block thrown across the mesh, about 2.4
        # cells in 100 steps, so that particles change cell all the time
        _plane("flow", "step", 160, 120, (0.1, 0.5, 0.25, 0.75), 200, E=1e5, nu=0.3, rho=1500.0, cfl=0.2,
               drift=0.12),
        # the package's scale-up workload (2.1M particles), a stretch of it
        _plane("scaleup_usf", "step", 1024, 1024, (0.0, 0.5, 0.0, 1.0), 100, cfl=0.025),
        # USL, 9 particles a cell, elastic beside fluid, an odd mesh
        _plane("step_usl_odd", "step", 701, 443, (0.13, 0.71, 0.0, 0.6), 60, side=3, scheme="usl",
               material="mixed", cfl=0.05),
        # the package's large mixed workload (16.8M particles, 4096 x 4096)
        _plane("mixed_large", "step", 4096, 4096, (0.125, 0.875, 0.0, 0.5), 30, scheme="usl",
               material="gap", E=5e6, nu=0.3, rho=1800.0, cfl=0.05),
        # one iteration of an inverse problem: the package's differentiation
        # workload (per-particle E, 125,664 particles), forward and backward
        _plane("grad_field", "autograd", 256, 256, (0.1, 0.9, 0.0, 0.6), 300, nu=0.3, rho=1000.0, cfl=0.05),
        # the same on a small odd mesh under USL, gradients in E, x0 and v0
        _plane("grad_usl", "adjoint", 150, 91, (0.12, 0.8, 0.0, 0.63), 120, scheme="usl", cfl=0.05,
               checkpoint=40),
        # many uneven simulations at once, as in the package's benchmark:
        # forward only, and forward with the adjoint
        _batch("batch_step", "batch", 64, 5, 100),
        _batch("batch_grad", "batch_grad", 40, 6, 200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve_loads", "line", "line_grad", "flow", "step", "step", "step",
                       "autograd", "adjoint", "batch", "batch_grad"])
    if kind == "line":
        return _pure(_bar("", kind, _log(rng, 5, 200), rng.randint(1, 5), _log(rng, 100, 500),
                          scheme=rng.choice(["usf", "usl"])))
    if kind == "line_grad":
        return _pure(_bar("", kind, _log(rng, 1, 40), rng.randint(1, 4), _log(rng, 100, 600),
                          scheme=rng.choice(["usf", "usl"]), E=1e4, dt=5e-4, gravity=0.0, force=0.0))
    if kind in ("batch", "batch_grad"):
        return _pure(_batch("", kind, _log(rng, 3, 48 if kind == "batch" else 24), rng.randint(0, 10 ** 6),
                            _log(rng, 40, 100), checkpoint=rng.choice([25, 50, 100])))
    x0 = rng.uniform(0.06, 0.3)
    y0 = rng.choice([0.0, 0.0, rng.uniform(0.05, 0.2)])
    box = (x0, x0 + rng.uniform(0.3, 0.6), y0, y0 + rng.uniform(0.3, 0.65))
    scheme = rng.choice(["usf", "usl"])
    mat = dict(material=rng.choice(["elastic", "mixed"]), E=10 ** rng.uniform(5, 7), nu=rng.uniform(0.2, 0.35),
               rho=rng.choice([1000.0, 1500.0, 2000.0]), cfl=rng.uniform(0.03, 0.06))
    if kind in ("solve", "solve_loads"):
        nx = _log(rng, 8, 128)
        return _pure(_plane("", kind, nx, max(6, int(nx * rng.uniform(0.5, 1.3))), box, _log(rng, 100, 500),
                            scheme=scheme, **mat))
    if kind == "flow":
        nx = _log(rng, 40, 300)
        mat.update(material="elastic", E=1e5, cfl=rng.uniform(0.1, 0.2))
        return _pure(_plane("", "step", nx, int(nx * rng.uniform(0.7, 1.1)), (0.1, 0.5, 0.25, 0.7),
                            _log(rng, 80, 200), drift=rng.uniform(0.03, 0.12),
                            velocity_update=rng.choice([False, True]), **mat))
    if kind == "step":
        nx = _log(rng, 64, 1200)
        return _pure(_plane("", "step", nx, int(nx * rng.uniform(0.5, 1.2)), box, _log(rng, 30, 120),
                            side=rng.choice([1, 2, 2, 2, 3]), scheme=scheme, reinit=rng.random() < 0.8, **mat))
    nx = _log(rng, 30, 260)
    return _pure(_plane("", kind, nx, int(nx * rng.uniform(0.5, 1.2)), box, _log(rng, 50, 200), scheme=scheme,
                        checkpoint=rng.choice([25, 50, 100]), **mat))


def _pure(c):
    c.pop("name")
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _cells(c):
    """Cell blocks (i0, i1, j0, j1, material) of a 2-D case, each at least one
    cell and inside the mesh."""
    i0, j0 = int(c["x0"] * c["nx"]), int(c["y0"] * c["ny"])
    i1 = min(c["nx"], max(i0 + 1, int(round(c["x1"] * c["nx"]))))
    j1 = min(c["ny"], max(j0 + 1, int(round(c["y1"] * c["ny"]))))
    if c["material"] == "elastic":
        return [(i0, i1, j0, j1, 0)]
    if c["material"] == "mixed":          # side by side
        im = (i0 + i1) // 2
        return [b for b in ((i0, im, j0, j1, 0), (im, i1, j0, j1, 1)) if b[1] > b[0]]
    third = (i1 - i0) // 3                # "gap": two blocks and nothing between them
    return [(i0, i0 + third, j0, j1, 0), (i1 - third, i1, j0, j1, 1)]


def _materials(c):
    m = [{"kind": "elastic", "density": c["rho"], "youngs_modulus": c["E"], "poisson_ratio": c["nu"]}]
    if c["material"] != "elastic":
        m.append({"kind": "newtonian", "density": 1000.0, "bulk_modulus": 2e6, "dynamic_viscosity": 1e-3})
    return m


def _wave(m):
    if m["kind"] == "newtonian":
        return math.sqrt(m["bulk_modulus"] / m["density"])
    E, nu = m["youngs_modulus"], m["poisson_ratio"]
    return math.sqrt(E * (1 - nu) / ((1 + nu) * (1 - 2 * nu)) / m["density"])


def _count(c):
    return sum((i1 - i0) * (j1 - j0) for i0, i1, j0, j1, _ in _cells(c)) * c["side"] ** 2


def _modes(x, size, amp, rnd):
    """Three seeded sine modes of each velocity component."""
    v = torch.zeros_like(x)
    for d in range(2):
        for _ in range(3):
            kx, ky, ph = rnd.uniform(0.5, 2.0), rnd.uniform(0.5, 2.0), rnd.uniform(0, 2 * math.pi)
            v[:, d] += amp * rnd.uniform(0.4, 1.0) * torch.sin(
                2 * math.pi * (kx * x[:, 0] + ky * x[:, 1]) / size + ph)
    return v


def _scene(c, seed):
    """Mesh, materials, loads and initial state of a 2-D case (float32 torch
    tensors on the GPU, the same for the same seed)."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(1000003 * seed + 17)
    rnd = random.Random(seed)
    nx, ny, side = c["nx"], c["ny"], c["side"]
    h = float(np.float32(c["size"] / nx))
    mats = _materials(c)
    cw = max(_wave(m) for m in mats)
    g = 1.0 / (2.0 * math.sqrt(3.0))
    off = {1: [0.5], 2: [0.5 - g, 0.5 + g], 3: [1 / 6, 0.5, 5 / 6]}[side]
    locs, mids = [], []
    for i0, i1, j0, j1, mid in _cells(c):
        off_x = torch.tensor(off, device=dev).repeat(side)
        off_y = torch.tensor(off, device=dev).repeat_interleave(side)
        px = torch.arange(i0, i1, device=dev)[None, :, None] + off_x
        py = torch.arange(j0, j1, device=dev)[:, None, None] + off_y
        p = torch.stack(torch.broadcast_tensors(px, py), -1).reshape(-1, 2)
        p += (torch.rand(p.shape, device=dev, generator=gen) - 0.5) * (0.2 if side < 3 else 0.1)
        locs.append(p)
        mids.append(torch.full((p.shape[0],), mid, dtype=torch.int32, device=dev))
    loc = (torch.cat(locs) * h).float()
    vel = _modes(loc, c["size"], c["amp"] * cw, rnd)
    vel += torch.tensor([c["drift"] * cw, 0.4 * c["drift"] * cw], device=dev)
    s = {"nx": nx, "ny": ny, "h": h, "dt": float(np.float32(c["cfl"] * h / cw)), "materials": mats,
         "scheme": c["scheme"], "reinit": c["reinit"], "velocity_update": c["velocity_update"],
         "loc": loc, "vel": vel.float(), "mid": torch.cat(mids), "E": None, "tractions": [], "nodal": []}
    I, J = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1))
    I, J = I.reshape(-1), J.reshape(-1)
    walls, bottom = np.nonzero((I == 0) | (I == nx))[0], np.nonzero(J == 0)[0]
    s["fixed"] = [(walls, 0), (bottom, 0), (bottom, 1)]
    if c["kind"] in ("autograd", "adjoint"):   # log-normal Young's modulus
        z = torch.randn(loc.shape[0], device=dev, generator=gen)
        s["E"] = (c["E"] * torch.exp(0.5 * z)).float()
    if c["kind"] == "solve_loads":
        i0, i1, j0, j1, _ = _cells(c)[0]
        top = torch.nonzero(loc[:, 1] > (j1 - 0.5) * h).reshape(-1)
        ramp = (0.0, 0.6 * c["steps"] * s["dt"])
        s["tractions"] = [(top.cpu().numpy(), 1, -0.01 * c["E"] * rnd.uniform(0.5, 1.0), ramp)]
        node = (j0 + j1) // 2 * (nx + 1) + i1    # a node on the block's right side
        s["nodal"] = [(np.array([node]), 0, 1e-3 * c["E"] * h * rnd.uniform(0.5, 1.0), ramp)]
    return s


def _target(c, s, seed):
    """Where an inverse problem wants the particles: a smooth displacement."""
    return (s["loc"] + _modes(s["loc"], c.get("size", 1.0), 0.01 * c.get("size", 1.0),
                              random.Random(seed + 99))).float()


def _spec(c, seed):
    """The members of a batch as 2-D cases: sizes from the case, moduli from
    the seed (0.05 m wide domains, rectangles of 20-60 %, as in the package's
    batching workload)."""
    size, mod, out = random.Random(c["spec"]), random.Random(seed), []
    for _ in range(c["members"]):
        n = size.randint(c["lo"], c["hi"])
        area, aspect = size.uniform(0.2, 0.6), math.exp(size.uniform(math.log(0.5), math.log(2.0)))
        w = min(0.9, math.sqrt(area * aspect))
        x0 = size.uniform(0.05, 0.95 - w)
        out.append(_plane("", "member", n, n, (x0, x0 + w, 0.0, min(0.9, area / w)), c["steps"],
                          E=math.exp(mod.uniform(math.log(1e5), math.log(1e8))), nu=mod.uniform(0.2, 0.35),
                          rho=1500.0, cfl=0.1, size=0.05))
    return out


def _bar_scene(c, seed):
    rnd = np.random.RandomState(seed)
    nx, ppe = c["nx"], c["ppe"]
    h = float(np.float32(1.0 / nx))
    last = max(1, int(0.9 * nx))          # elements [0, last) hold particles
    x = ((np.arange(last)[:, None] + (np.arange(ppe) + 0.5) / ppe) * h).reshape(-1)
    x = (x + rnd.uniform(-0.1, 0.1, x.size) * h / ppe).astype(np.float32)
    v = (c["v0"] * (1 + 0.2 * rnd.rand()) * np.sin(0.5 * np.pi * (x + 0.2 * rnd.rand()))).astype(np.float32)
    return {"nx": nx, "h": h, "dt": float(np.float32(c["dt"])), "loc": x, "vel": v, "last": last,
            "scheme": c["scheme"], "E": c["E"] * (1 + 0.1 * rnd.rand()), "rho": c["rho"],
            "force": c["force"], "ramp": (0.0, c["steps"] * c["dt"]), "gravity": c["gravity"]}


# ---------------------------------------------------------------------------
# the package's objects for them
# ---------------------------------------------------------------------------
def _material(m):
    props = {k: v for k, v in m.items() if k != "kind"}
    return {"elastic": D.LinearElastic, "newtonian": D.Newtonian}[m["kind"]](props)


def _solver(c, s):
    """The case through the object model (host arrays)."""
    n = s["loc"].shape[0]
    ramps = {}

    def ramp(r):
        return ramps.setdefault(r, D.Linear(len(ramps), np.array(r), np.array([0.0, 1.0])))

    el = D.Quadrilateral4Node(
        (s["nx"], s["ny"]), s["nx"] * s["ny"], (s["h"], s["h"]),
        [(ids, D.Constraint(d, 0.0)) for ids, d in s["fixed"]],
        concentrated_nodal_forces=[D.NodalForce(ids, ramp(r), d, f) for ids, d, f, r in s["nodal"]])
    ps = D.Particles(s["loc"].cpu().numpy().reshape(n, 1, 2), [_material(m) for m in s["materials"]],
                     np.zeros(n, np.int32), material_ids=s["mid"].cpu().numpy(),
                     youngs_modulus=None if s["E"] is None else s["E"].cpu().numpy())
    ps.velocity[:] = s["vel"].cpu().numpy().reshape(n, 1, 2)
    mesh = D.Mesh2D({"particles": [ps], "elements": el, "particle_surface_traction": [
        D.ParticleTraction(0, ids, ramp(r), d, f) for ids, d, f, r in s["tractions"]]})
    return D.MPMExplicit(mesh, s["dt"], scheme=s["scheme"], velocity_update=s["velocity_update"],
                         sim_steps=c["steps"])


def _bar_solver(c, s, E):
    cls, props = (D.SimpleMaterial, {"density": s["rho"], "E": s["E"]}) if c["kind"] == "line_grad" else (
        D.LinearElastic, {"density": s["rho"], "youngs_modulus": s["E"], "poisson_ratio": 0.3})
    forces = []
    if s["force"]:
        fn = D.Linear(0, np.array(s["ramp"]), np.array([0.0, 1.0]))
        forces = [D.NodalForce(np.array([s["last"]]), fn, 0, s["force"])]
    el = D.Linear1D(s["nx"], s["nx"], s["h"], [(np.array([0]), D.Constraint(0, 0.0))],
                    concentrated_nodal_forces=forces)
    n = s["loc"].size
    ps = D.Particles(s["loc"].reshape(n, 1, 1), cls(props), np.zeros(n, np.int32), youngs_modulus=E)
    ps.velocity[:] = s["vel"].reshape(n, 1, 1)
    mesh = D.Mesh1D({"particles": [ps], "elements": el, "particle_surface_traction": []})
    return D.MPMExplicit(mesh, s["dt"], scheme=s["scheme"], sim_steps=c["steps"])


def _simulation(s):
    """The case as one engine simulation with device arrays."""
    sim = D.Simulation((s["nx"], s["ny"]), (s["h"], s["h"]), s["dt"], scheme=s["scheme"],
                       velocity_update=s["velocity_update"], reinit_each_step=s["reinit"], gravity=GRAVITY,
                       constraints=[(ids, D.Constraint(d, 0.0)) for ids, d in s["fixed"]],
                       materials=[_material(m) for m in s["materials"]])
    sim.set_particles(s["loc"].contiguous(), s["mid"])
    sim.write("velocity", s["vel"].contiguous())
    if s["E"] is not None:
        sim.write("youngs_modulus", s["E"])
    sim.initialize()
    return sim


def _initial(s):
    """The initial value of every particle field, as device arrays."""
    n, dev = s["loc"].shape[0], s["loc"].device
    rho = torch.tensor([m["density"] for m in s["materials"]], dtype=torch.float32, device=dev)
    zero = torch.zeros((n, 6), device=dev)
    return {"loc": s["loc"].contiguous(), "velocity": s["vel"].contiguous(), "stress": zero, "strain": zero,
            "density": rho[s["mid"].long()].contiguous(), "volumetric_strain_centroid": torch.zeros(n, device=dev)}


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "line":
        return {"case": c, "solver": _bar_solver(c, _bar_scene(c, seed), None)}
    if kind == "line_grad":
        s = _bar_scene(c, seed)
        n = s["loc"].size
        return {"case": c, "solver": _bar_solver(c, s, np.full(n, s["E"])),
                "E": torch.tensor(s["E"], dtype=torch.float32, requires_grad=True), "n": n}
    if kind in ("solve", "solve_loads"):
        return {"case": c, "solver": _solver(c, _scene(c, seed))}
    if kind in ("step", "adjoint"):
        s = _scene(c, seed)
        n, dev = s["loc"].shape[0], s["loc"].device
        st = {"case": c, "sim": _simulation(s), "init": _initial(s),
              "nodal": torch.zeros(((c["nx"] + 1) * (c["ny"] + 1), 2), device=dev),
              "out": {k: torch.empty((n, 2 if k in ("loc", "velocity") else 6), device=dev) for k in RESULT}}
        if kind == "adjoint":
            st["target"] = _target(c, s, seed)
        return st
    if kind == "autograd":
        s = _scene(c, seed)
        return {"case": c, "solver": _solver(c, s), "E": s["E"].requires_grad_(), "target": _target(c, s, seed)}
    scenes = [_scene(m, seed + 7 * k) for k, m in enumerate(_spec(c, seed))]
    sims = [_simulation(s) for s in scenes]
    init = [_initial(s) for s in scenes]
    st = {"case": c, "sims": sims, "batch": D.Batch(sims), "counts": [s["loc"].shape[0] for s in scenes],
          "init": {k: torch.cat([i[k].reshape(-1) for i in init]) for k in STATE}}
    dev = st["init"]["loc"].device
    st["nodal"] = torch.zeros(sum(2 * s.nnodes for s in sims), device=dev)
    st["out"] = {k: torch.empty(sum(st["counts"]) * (2 if k in ("loc", "velocity") else 6), device=dev)
                 for k in RESULT}
    if kind == "batch_grad":
        st["target"] = torch.cat([_target({"size": 0.05}, s, seed).reshape(-1) for s in scenes])
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind in ("solve", "solve_loads"):
        return state["solver"].solve_jit(np.array(GRAVITY))
    if kind == "line":
        return state["solver"].solve_jit(np.array([c["gravity"]]))
    if kind == "line_grad":
        E = state["E"]
        x, v = explicit_run(state["solver"], [c["gravity"]], E.expand(state["n"]), nsteps=c["steps"])
        loss = ((v - 0.05) ** 2).sum() + (x ** 2).sum()
        (grad,) = torch.autograd.grad(loss, E)
        return {"loc": x.detach(), "velocity": v.detach(), "grad": grad}
    if kind == "autograd":
        E, n = state["E"], state["E"].shape[0]
        x, v = explicit_run(state["solver"], GRAVITY, E, checkpoint_steps=c["checkpoint"])
        loss = ((x - state["target"]) ** 2).sum(1).mean() * n
        (grad,) = torch.autograd.grad(loss, E)
        return {"loc": x.detach(), "velocity": v.detach(), "grad": grad}
    if kind in ("step", "adjoint"):
        sim, out = state["sim"], state["out"]
        for k in STATE:
            sim.write(k, state["init"][k])
        sim.write_nodal("velocity", state["nodal"])
        sim.step_index = 0
        sim.initialize()
        if kind == "step":
            sim.step(c["steps"])
            return {k: sim.read(k, out=out[k]) for k in RESULT}
        sim.record(c["steps"], checkpoint_steps=c["checkpoint"])
        x = sim.read("loc", out=out["loc"])
        v = sim.read("velocity", out=out["velocity"])
        g = sim.adjoint(2.0 * (x - state["target"]), 0.1 * v)
        return {"loc": x, "velocity": v, "grad": g["youngs_modulus"], "grad_loc": g["loc"],
                "grad_velocity": g["velocity"]}
    b, out = state["batch"], state["out"]
    for k in STATE:
        b.write(k, state["init"][k])
    b.write_nodal("velocity", state["nodal"])
    b.restart()
    if kind == "batch":
        b.step(c["steps"])
        return {k: b.read(k, out=out[k]) for k in RESULT}
    b.record(c["steps"], checkpoint_steps=c["checkpoint"])
    x = b.read("loc", out=out["loc"])
    seeds = (2.0 * (x - state["target"])).split([2 * n for n in state["counts"]])
    g = b.adjoint([t.view(-1, 2) for t in seeds], want=("youngs_modulus",))
    return {"loc": x, "grad": torch.cat([m["youngs_modulus"] for m in g])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes and operations of a pass.  A forward step reads and writes each
    particle's state once (x, v, stress, strain, density, volumetric strain:
    13 floats) and touches 72 B a node; about 330 operations a particle.  A
    reverse step reads the step's particle state and nodal results (9 floats a
    particle, 7 a node) and reads and writes the ten adjoints it carries;
    about 600 operations a particle, and the forward state is kept once."""
    c, kind = case, case["kind"]
    if kind in ("line", "line_grad"):
        n, nn = max(1, int(0.9 * c["nx"])) * c["ppe"], c["nx"] + 1
        k = c["steps"] * (2 if kind == "line_grad" else 1)
        return {"bytes": float(k * (104 * n + 20 * nn)), "flops": float(k * 120 * n)}
    if kind in ("batch", "batch_grad"):
        members = _spec(c, 0)
        n, nn = sum(_count(m) for m in members), sum((m["nx"] + 1) * (m["ny"] + 1) for m in members)
    else:
        n, nn = _count(c), (c["nx"] + 1) * (c["ny"] + 1)
    by, fl = 104.0 * n + 72.0 * nn, 330.0 * n
    if kind in ("autograd", "adjoint", "batch_grad"):
        by += (36 + 36 + 80) * n + (28 + 28) * nn
        fl += 600.0 * n
    return {"bytes": by * c["steps"], "flops": fl * c["steps"]}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _flush(a):
    return torch.where(a.abs() < FLUSH, torch.zeros_like(a), a)


class _Exact:
    """The explicit step of one or several 2-D scenes side by side, float64."""

    def __init__(self, scenes):
        f, dev = torch.float64, scenes[0]["loc"].device
        self.dev, s0 = dev, scenes[0]
        self.scheme, self.reinit, self.pic = s0["scheme"], s0["reinit"], s0["velocity_update"]
        counts = [s["loc"].shape[0] for s in scenes]

        def each(values, dtype=f):   # a value per scene as one per particle (or a scalar)
            if len(scenes) == 1:
                return torch.tensor(values[0], dtype=dtype, device=dev)
            return torch.repeat_interleave(torch.tensor(values, dtype=dtype, device=dev),
                                           torch.tensor(counts, device=dev))

        nns = [(s["nx"] + 1) * (s["ny"] + 1) for s in scenes]
        ncs = [s["nx"] * s["ny"] for s in scenes]
        self.nn, self.nc = sum(nns), sum(ncs)
        self.nx = each([s["nx"] for s in scenes], torch.long)
        self.node0 = each([sum(nns[:k]) for k in range(len(scenes))], torch.long)
        self.cell0 = each([sum(ncs[:k]) for k in range(len(scenes))], torch.long)
        self.h, self.dt = each([s["h"] for s in scenes]), each([s["dt"] for s in scenes])
        nodes = torch.tensor(nns, device=dev)
        self.node_dt = torch.repeat_interleave(torch.tensor([s["dt"] for s in scenes], dtype=f, device=dev), nodes)
        self.free = torch.ones(self.nn, 2, dtype=torch.bool, device=dev)
        at = 0
        for s, k in zip(scenes, nns):
            for ids, d in s["fixed"]:
                self.free[at + torch.as_tensor(ids, device=dev), d] = False
            at += k
        mid = torch.cat([s["mid"] for s in scenes]).long()
        table = [s["materials"] for s in scenes]
        self.newton = torch.zeros(mid.shape[0], dtype=torch.bool, device=dev)
        par = {k: torch.zeros(mid.shape[0], dtype=f, device=dev) for k in ("E", "nu", "K", "mu", "rho")}
        at = 0
        for mats, k in zip(table, counts):
            sl = mid[at:at + k]
            for i, m in enumerate(mats):
                p = sl == i
                par["rho"][at:at + k][p] = m["density"]
                if m["kind"] == "newtonian":
                    self.newton[at:at + k][p] = True
                    par["K"][at:at + k][p], par["mu"][at:at + k][p] = m["bulk_modulus"], m["dynamic_viscosity"]
                else:
                    par["E"][at:at + k][p], par["nu"][at:at + k][p] = m["youngs_modulus"], m["poisson_ratio"]
            at += k
        self.fluid = bool(self.newton.any())
        self.K, self.mu, nu = par["K"], par["mu"], par["nu"]
        bulk, shear = 1 / (3 * (1 - 2 * nu)), 1 / (2 * (1 + nu))
        self.c1, self.c2, self.c3 = bulk + 4 * shear / 3, bulk - 2 * shear / 3, shear
        self.E = par["E"] if s0["E"] is None else torch.cat([s["E"] for s in scenes]).detach().double()
        self.tractions, self.nodal = s0["tractions"], s0["nodal"]
        n = mid.shape[0]
        self.start = {"x": torch.cat([s["loc"] for s in scenes]).double(),
                      "v": torch.cat([s["vel"] for s in scenes]).double(),
                      "sig": torch.zeros(n, 4, dtype=f, device=dev), "eps": torch.zeros(n, 3, dtype=f, device=dev),
                      "rho": par["rho"].clone(), "vsc": torch.zeros(n, dtype=f, device=dev),
                      "nv": torch.zeros(self.nn, 2, dtype=f, device=dev)}
        if not self.reinit:
            cell = self._cells(self.start["x"])[2]
            cnt = torch.bincount(cell, minlength=self.nc)[cell]
            vol = (self.h * self.h / cnt).expand(n)
            self.start["vol"], self.start["mass"] = vol.clone(), vol * par["rho"]

    def _cells(self, x):
        with torch.no_grad():
            i = torch.floor(x[:, 0] / self.h).long()
            j = torch.floor(x[:, 1] / self.h).long()
        return i, j, self.cell0 + j * self.nx + i

    def _nodes(self, ids, terms):
        out = torch.zeros(self.nn, dtype=torch.float64, device=self.dev)
        for k in range(4):
            out = out.index_add(0, ids[k], terms[k])
        return out

    def _stress(self, st, E, G, Gc, ids, nv):
        """Strain, volumetric strain and stress after the rates of ``nv``."""
        vx, vy = [nv[i, 0] for i in ids], [nv[i, 1] for i in ids]

        def dot(a, b):
            return sum(p * q for p, q in zip(a, b))

        r0, r1 = _flush(dot(G[0], vx)), _flush(dot(G[1], vy))
        r3 = _flush(dot(G[0], vy) + dot(G[1], vx))
        dvol = self.dt * (_flush(dot(Gc[0], vx)) + _flush(dot(Gc[1], vy)))
        d0, d1, d3 = r0 * self.dt, r1 * self.dt, r3 * self.dt
        vsc, s = st["vsc"] + dvol, st["sig"]
        a1, a2 = E * self.c1, E * self.c2
        sig = s + torch.stack([a1 * d0 + a2 * d1, a2 * d0 + a1 * d1, a2 * (d0 + d1), E * self.c3 * d3], 1)
        if self.fluid:
            kv, t3 = self.K * vsc, (r0 + r1) / 3
            tot = torch.stack([kv + 2 * self.mu * (r0 - t3), kv + 2 * self.mu * (r1 - t3),
                               kv - 2 * self.mu * t3, self.mu * r3], 1)
            sig = torch.where(self.newton[:, None], tot, sig)
        return {"sig": sig, "eps": st["eps"] + torch.stack([d0, d1, d3], 1), "vsc": vsc,
                "rho": st["rho"] / (1 + dvol)}, dvol

    def step(self, st, t, E=None):
        E = self.E if E is None else E
        x, v = st["x"], st["v"]
        i, j, cell = self._cells(x)
        r = 2 / self.h
        xi, eta = (x[:, 0] - (i + 0.5) * self.h) * r, (x[:, 1] - (j + 0.5) * self.h) * r
        ll = self.node0 + j * (self.nx + 1) + i
        ids = [ll, ll + 1, ll + self.nx + 2, ll + self.nx + 1]
        sx, sy = (-1, 1, 1, -1), (-1, -1, 1, 1)
        N = [0.25 * (1 + sx[k] * xi) * (1 + sy[k] * eta) for k in range(4)]
        G = ([0.25 * sx[k] * (1 + sy[k] * eta) * r for k in range(4)],
             [0.25 * sy[k] * (1 + sx[k] * xi) * r for k in range(4)])
        Gc = ([0.25 * sx[k] * r for k in range(4)], [0.25 * sy[k] * r for k in range(4)])
        if self.reinit:
            V0 = self.h * self.h / torch.bincount(cell, minlength=self.nc)[cell]
            m = V0 * st["rho"]
        else:
            V0, m = st["vol"], st["mass"]
        M = self._nodes(ids, [m * n for n in N])
        some = (M != 0)[:, None]
        inv = torch.where(M == 0, torch.ones_like(M), M)[:, None]
        P = torch.stack([self._nodes(ids, [n * (m * v[:, d]) for n in N]) for d in range(2)], 1)
        nv = torch.where(self.free, _flush(torch.where(some, _flush(P) / inv, st["nv"].detach())), 0.0)
        new, V = {}, V0
        if self.scheme == "usf":
            new, dvol = self._stress(st, E, G, Gc, ids, nv)
            V = V0 * (1 + dvol)
        s = new.get("sig", st["sig"])
        sxx, syy, sxy = s[:, 0], s[:, 1], s[:, 3]
        f = [[], []]
        pull = [torch.zeros_like(V), torch.zeros_like(V)]
        for pids, d, value, ramp in self.tractions:
            at = min(1.0, t * float(self.dt) / ramp[1])
            pids = torch.as_tensor(pids, device=self.dev)
            size = torch.sqrt(V0[pids])
            pull[d] = pull[d].index_add(0, pids, at * value * V[pids] / size)
        for k in range(4):
            f[0].append(N[k] * (m * GRAVITY[0] + pull[0]) - V * (G[0][k] * sxx + G[1][k] * sxy))
            f[1].append(N[k] * (m * GRAVITY[1] + pull[1]) - V * (G[1][k] * syy + G[0][k] * sxy))
        F = torch.stack([self._nodes(ids, f[0]), self._nodes(ids, f[1])], 1)
        for nids, d, value, ramp in self.nodal:
            F[torch.as_tensor(nids, device=self.dev), d] += min(1.0, t * float(self.dt) / ramp[1]) * value
        a = torch.where(some, F / inv, 0.0)
        nb = _flush(torch.where(self.free, nv + a * self.node_dt[:, None], 0.0))
        a = _flush(torch.where(self.free, a, 0.0))
        vh = sum(n[:, None] * nb[i] for n, i in zip(N, ids))
        ah = sum(n[:, None] * a[i] for n, i in zip(N, ids))
        dt = self.dt[:, None] if self.dt.dim() else self.dt
        if self.scheme == "usl":
            new, dvol = self._stress(st, E, G, Gc, ids, nb)
            V = V0 * (1 + dvol)
        new.update(x=x + vh * dt, v=vh if self.pic else v + ah * dt, nv=nb)
        if not self.reinit:
            new.update(vol=V, mass=m)
        return new

    def run(self, steps, keep=False):
        st, kept = self.start, []
        with torch.no_grad():
            for t in range(steps):
                if keep:
                    kept.append(st)
                st = self.step(st, t)
        return st, kept

    def reverse(self, kept, gx, gv):
        """Adjoints of E and of the start's x and v for those of the end."""
        names = ("x", "v", "sig", "rho", "vsc")
        adj = {"x": gx, "v": gv, **{k: torch.zeros_like(kept[0][k]) for k in names[2:]}}
        E, gE = self.E.clone().requires_grad_(), torch.zeros_like(self.E)
        for t in range(len(kept) - 1, -1, -1):
            st = {k: (a.detach().requires_grad_() if k in names else a) for k, a in kept[t].items()}
            new = self.step(st, t, E)
            got = torch.autograd.grad([new[k] for k in names], [E] + [st[k] for k in names],
                                      [adj[k] for k in names], allow_unused=True)
            gE += got[0]
            adj = {k: torch.zeros_like(st[k]) if g is None else g for k, g in zip(names, got[1:])}
        return gE, adj["x"], adj["v"]


def _fields(st):
    s, e = st["sig"], st["eps"]
    z = torch.zeros_like(s[:, 0])
    return {"loc": st["x"], "velocity": st["v"],
            "stress": torch.stack([s[:, 0], s[:, 1], s[:, 2], s[:, 3], z, z], 1),
            "strain": torch.stack([e[:, 0], e[:, 1], z, e[:, 2], z, z], 1)}


def _bar_step(s, simple, st, t, E, dev):
    """One step of the bar in float64."""
    h, dt, nx = s["h"], s["dt"], s["nx"]
    x, v = st["x"], st["v"]
    with torch.no_grad():
        e = torch.floor(x / h).long()
    xi = (x - (e + 0.5) * h) * (2 / h)
    N, dN = [0.5 * (1 - xi), 0.5 * (1 + xi)], [-1 / h, 1 / h]
    V0 = h / torch.bincount(e, minlength=nx)[e]
    m = V0 * st["rho"]

    def nodes(terms):
        out = torch.zeros(nx + 1, dtype=torch.float64, device=dev)
        return out.index_add(0, e, terms[0]).index_add(0, e + 1, terms[1])

    def update(nv):
        r = _flush(dN[0] * nv[e] + dN[1] * nv[e + 1])
        d = r * dt
        if simple:
            sig = st["sig"] + torch.stack([E * d, 0 * d, 0 * d], 1)
        else:
            k, g = 1 / (3 * 0.4), 1 / 2.6      # Poisson's ratio 0.3
            a1, a2 = E * (k + 4 * g / 3), E * (k - 2 * g / 3)
            sig = st["sig"] + torch.stack([a1 * d, a2 * d, a2 * d], 1)
        return {"sig": sig, "eps": st["eps"] + d, "rho": st["rho"] / (1 + d)}, V0 * (1 + d)

    free = torch.ones(nx + 1, dtype=torch.bool, device=dev)
    free[0] = False
    M, P = nodes([m * n for n in N]), _flush(nodes([n * (m * v) for n in N]))
    inv = torch.where(M == 0, torch.ones_like(M), M)
    nv = torch.where(free, _flush(torch.where(M == 0, st["nv"].detach(), P / inv)), 0.0)
    new, V = update(nv) if s["scheme"] == "usf" else ({}, V0)
    sxx = new.get("sig", st["sig"])[:, 0]
    F = nodes([n * m * s["gravity"] - V * sxx * d for n, d in zip(N, dN)])
    if s["force"]:
        F[s["last"]] += min(1.0, t * dt / s["ramp"][1]) * s["force"]
    a = torch.where(M == 0, torch.zeros_like(F), F / inv)
    nb, a = _flush(torch.where(free, nv + a * dt, 0.0)), _flush(torch.where(free, a, 0.0))
    if s["scheme"] == "usl":
        new, _ = update(nb)
    new.update(x=x + (N[0] * nb[e] + N[1] * nb[e + 1]) * dt, v=v + (N[0] * a[e] + N[1] * a[e + 1]) * dt, nv=nb)
    return new


def _bar_exact(c, seed):
    s, dev, f = _bar_scene(c, seed), _device(), torch.float64
    n, simple = s["loc"].size, c["kind"] == "line_grad"
    st = {"x": torch.tensor(s["loc"], dtype=f, device=dev), "v": torch.tensor(s["vel"], dtype=f, device=dev),
          "sig": torch.zeros(n, 3, dtype=f, device=dev), "eps": torch.zeros(n, dtype=f, device=dev),
          "rho": torch.full((n,), s["rho"], dtype=f, device=dev),
          "nv": torch.zeros(s["nx"] + 1, dtype=f, device=dev)}
    E0 = float(np.float32(s["E"])) if simple else s["E"]
    E = torch.tensor(E0, dtype=f, device=dev, requires_grad=simple)
    with torch.set_grad_enabled(simple):
        for t in range(c["steps"]):
            st = _bar_step(s, simple, st, t, E, dev)
        if simple:
            loss = ((st["v"] - 0.05) ** 2).sum() + (st["x"] ** 2).sum()
            (grad,) = torch.autograd.grad(loss, E)
            return {"loc": st["x"].detach()[:, None], "velocity": st["v"].detach()[:, None], "grad": grad}
    z = torch.zeros(n, 3, dtype=f, device=dev)
    return {"loc": st["x"], "velocity": st["v"], "stress": torch.cat([st["sig"], z], 1),
            "strain": torch.cat([st["eps"][:, None], z, z[:, :2]], 1)}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("line", "line_grad"):
        return _bar_exact(c, seed)
    if kind in ("batch", "batch_grad"):
        scenes = [_scene(m, seed + 7 * k) for k, m in enumerate(_spec(c, seed))]
        ex = _Exact(scenes)
        end, kept = ex.run(c["steps"], keep=kind == "batch_grad")
        if kind == "batch":
            return {k: a.reshape(-1) for k, a in _fields(end).items()}
        target = torch.cat([_target({"size": 0.05}, s, seed) for s in scenes]).double()
        gE, _, _ = ex.reverse(kept, 2 * (end["x"] - target), torch.zeros_like(end["v"]))
        return {"loc": end["x"].reshape(-1), "grad": gE}
    s = _scene(c, seed)
    ex = _Exact([s])
    if kind in ("autograd", "adjoint"):
        end, kept = ex.run(c["steps"], keep=True)
        gx = 2 * (end["x"] - _target(c, s, seed).double())
        gv = 0.1 * end["v"] if kind == "adjoint" else torch.zeros_like(end["v"])
        gE, g0, gv0 = ex.reverse(kept, gx, gv)
        out = {"loc": end["x"], "velocity": end["v"], "grad": gE}
        return out if kind == "autograd" else {**out, "grad_loc": g0, "grad_velocity": gv0}
    return _fields(ex.run(c["steps"])[0])
