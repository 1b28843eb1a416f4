"""Steps in one cooperative launch (k_steps_resident), taken when every listed
tile has an SM of its own, leave the state that one launch a phase leaves, bit
for bit: over meshes of one tile, of part of a wave, of the last whole wave, and
of more tiles than SMs of which few or many are active; step counts around the
shortest resident sequence; schemes, volume set-ups, loads, drift and
rolled-back blocks."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

FIELDS = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid", "volume", "mass",
          "element_ids")
# cells of the mesh, cells of the filled block (a tile owns 31 x 15 nodes)
MESHES = {
    "one-tile": ((20, 12), (4, 10, 3, 8)),
    "twenty-five": ((140, 65), (5, 120, 4, 60)),
    "wave": ((247, 278), (10, 200, 5, 150)),          # 8 x 19 = 152 tiles
    "few-active": ((371, 194), (100, 160, 60, 100)),  # 12 x 13 = 156 tiles
    "all-active": ((371, 194), (2, 350, 2, 190)),     # one launch a phase
}
RUNS = {
    "usf": dict(),
    "usl": dict(scheme="usl"),
    "solve-usf-newtonian": dict(reinit=False, newtonian=True),
    "solve-usl-loads": dict(reinit=False, scheme="usl", loads=True),
    "usf-loads": dict(loads=True, newtonian=True),
    "usf-fast": dict(speed=6.0),                      # drifts: re-sorts between blocks
    "usl-thrown": dict(speed=40.0, scheme="usl"),     # two cells in a block: rolled back
}


def make(mesh, scheme="usf", reinit=True, newtonian=False, loads=False, speed=0.0, one_launch_a_phase=False):
    (nx, ny), (i0, i1, j0, j1) = MESHES[mesh]
    rng = np.random.Generator(np.random.PCG64(11))
    h = 1.0 / 128
    mats = [D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3})]
    if newtonian:
        mats.append(D.Newtonian({"density": 900.0, "bulk_modulus": 1e5, "dynamic_viscosity": 1e-2}))
    ramp = D.Linear(0, np.array([0.0, 2e-3]), np.array([0.0, 1.0]))
    bottom = np.arange(nx + 1)
    sim = D.Simulation((nx, ny), (h, h), 4e-5, scheme=scheme, reinit_each_step=reinit, gravity=(0.5, -9.81),
                       materials=mats, functions=[ramp],
                       constraints=[(bottom, D.Constraint(0, 0.0)), (bottom, D.Constraint(1, 0.0))],
                       nodal_forces=[D.NodalForce(np.array([4 * (nx + 1) + 5]), ramp, 0, 3.0)] if loads else [])
    i, j = np.meshgrid(np.arange(i0, i1), np.arange(j0, j1))
    off = np.array([0.25, 0.75])
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    loc = (np.stack([x, y], 1) + rng.uniform(-0.1, 0.1, (x.size, 2))) * h
    n = len(loc)
    vel = np.stack([speed + np.sin(40 * loc[:, 1]), 0.3 * np.cos(30 * loc[:, 0])], 1)
    sim.set_particles(loc.astype(np.float32), (rng.permutation(n) % 3 == 0).astype(np.int32) * int(newtonian))
    sim.write("velocity", vel.astype(np.float32))
    if loads:
        pid = np.arange(0, n, 7)
        sim.set_tractions(pid, np.ones(pid.size, np.int32), np.full(pid.size, -50.0), [ramp] * pid.size)
        sim.set_particle_velocity_constraints([n // 2], [0], [0.1])
    if one_launch_a_phase:
        sim.set_kernel_variant(forces_lpc=2)          # documented: the same results
    sim.set_block_steps(24)
    sim.initialize()
    return sim


@pytest.mark.parametrize("name", list(RUNS))
@pytest.mark.parametrize("mesh", list(MESHES))
def test_resident_steps_equal_launches(built, mesh, name):
    run = dict(RUNS[name])
    if mesh == "one-tile" and run.get("speed"):
        run["speed"] = min(run["speed"], 15.0)        # 61 steps stay inside 20 cells
    a, b = make(mesh, **run), make(mesh, one_launch_a_phase=True, **run)
    for n in (1, 7, 8, 9, 36):                        # 36: blocks of 24 and 12
        a.step(n)
        b.step(n)
        for f in FIELDS:
            assert np.array_equal(a.read(f), b.read(f)), (f, n)
        for f in ("mass", "velocity", "acceleration"):
            assert np.array_equal(a.read_nodal(f), b.read_nodal(f)), (f, n)
    assert a.counters() == b.counters()
    assert a.step_index == b.step_index == 61
    if name == "usf-fast" and mesh != "one-tile":
        assert a.counters()["resorts"] > 1
