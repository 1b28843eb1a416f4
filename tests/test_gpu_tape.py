"""The tape of a recorded run (csrc/mpm_adjoint.cu): taped steps leave the state
that plain steps leave, and the gradients of a run kept whole are those of the
same run kept as checkpoints and re-run, bit for bit -- over schemes, volume
set-ups, materials, loads, re-sorts and rolled-back blocks, for one simulation
and for batches, and when the same handle records again (its second recording
goes through captured graphs)."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

FIELDS = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid", "volume", "mass",
          "element_ids")
CASES = {
    "usf": dict(),
    "usl-split": dict(scheme="usl", split=0),
    "solve-usf-newtonian": dict(reinit=False, newtonian=True, split=0),
    "solve-usl": dict(reinit=False, scheme="usl"),
    "usf-loads": dict(loads=True, newtonian=True),
    "usl-fast": dict(scheme="usl", speed=8.0, split=0),      # re-sorts between blocks
    "usf-thrown": dict(speed=40.0, split=0),                 # two cells in a block: rolled back
    "pic": dict(velocity_update=True, newtonian=True, scheme="usl"),
}


def make(nx=70, ny=50, scheme="usf", reinit=True, newtonian=False, loads=False, speed=0.0, split=None,
         velocity_update=False, seed=3):
    rng = np.random.Generator(np.random.PCG64(seed))
    h = 1.0 / 128
    mats = [D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3})]
    if newtonian:
        mats.append(D.Newtonian({"density": 900.0, "bulk_modulus": 1e5, "dynamic_viscosity": 1e-2}))
    ramp = D.Linear(0, np.array([0.0, 2e-3]), np.array([0.0, 1.0]))
    bottom = np.arange(nx + 1)
    sim = D.Simulation((nx, ny), (h, h), 4e-5, scheme=scheme, reinit_each_step=reinit, gravity=(0.5, -9.81),
                       velocity_update=velocity_update, materials=mats, functions=[ramp],
                       constraints=[(bottom, D.Constraint(0, 0.0)), (bottom, D.Constraint(1, 0.0))],
                       nodal_forces=[D.NodalForce(np.array([12 * (nx + 1) + 20]), ramp, 0, 3.0)] if loads else [])
    if split is not None:
        sim.set_empty_split(split)
    i, j = np.meshgrid(np.arange(8, 28), np.arange(6, 20))
    off = np.array([0.25, 0.75])
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    loc = (np.stack([x, y], 1) + rng.uniform(-0.1, 0.1, (x.size, 2))) * h
    n = len(loc)
    vel = np.stack([speed + np.sin(40 * loc[:, 1]), 0.3 * np.cos(30 * loc[:, 0])], 1)
    E = 1e5 * np.exp(rng.uniform(-0.5, 0.5, n))
    mid = (rng.permutation(n) % 3 == 0).astype(np.int32) * int(newtonian)

    def start():
        sim.set_particles(loc.astype(np.float32), mid)
        sim.write("velocity", vel.astype(np.float32))
        sim.write("youngs_modulus", E.astype(np.float32))
        if loads:
            pid = np.arange(0, n, 7)
            sim.set_tractions(pid, np.ones(pid.size, np.int32), np.full(pid.size, -50.0), [ramp] * pid.size)
            sim.set_particle_velocity_constraints([n // 2], [0], [0.1])
        sim.set_block_steps(24)
        sim.initialize()

    start()
    return sim, start, rng.standard_normal((4, n, 2)).astype(np.float32)


def gradients(sim, w):
    a = sim.adjoint(w[0], w[1])
    sim.read("volume")                      # may re-sort; the recording does not depend on it
    b = sim.adjoint(w[2], w[3])             # the same recording, other seeds
    return {**{"1 " + k: v for k, v in a.items()}, **{"2 " + k: v for k, v in b.items()}}


@pytest.mark.parametrize("K", [100, 7, 30, 61])
@pytest.mark.parametrize("name", list(CASES))
def test_whole_tape_equals_checkpoints(built, name, K):
    steps = 61
    sim, _, _ = make(**CASES[name])
    for done in range(0, steps, K):         # a recording's blocks end at its checkpoints
        sim.step(min(K, steps - done))
    counters = sim.counters()
    plain = {f: sim.read(f) for f in FIELDS}
    nodal = {f: sim.read_nodal(f) for f in ("mass", "velocity", "acceleration")}
    ref = None
    for limit in (-1, 0):
        sim, start, w = make(**CASES[name])
        sim.set_tape_limit(limit)
        for again in range(2):
            if again:
                start()
            sim.record(steps, K)
            if not again:
                assert sim.counters() == counters, limit
            for f in FIELDS:
                assert np.array_equal(sim.read(f), plain[f], equal_nan=True), (limit, f)
            for f in nodal:
                assert np.array_equal(sim.read_nodal(f), nodal[f]), (limit, f)
            g = gradients(sim, w)
            ref = ref or g
            for k in g:
                assert np.isfinite(g[k]).all() and np.array_equal(g[k], ref[k]), (limit, again, k)
    if name == "usf-thrown" and K > 20:
        assert counters["rollbacks"] > 0
    if name == "usl-fast":
        assert counters["resorts"] > 1


@pytest.mark.parametrize("names", [("usf", "usf-thrown"), ("usl-split", "usl-fast"),
                                   ("solve-usf-newtonian",), ("usf-loads",)])
def test_batched_tape_equals_single(built, names):
    steps, K = 61, 20
    cases = [dict(CASES[n], seed=5 + i, nx=70 + 9 * i, ny=50 - 4 * i) for i, n in enumerate(names)]
    refs = []
    for c in cases:
        sim, _, w = make(**c)
        sim.record(steps, K)
        refs.append(({f: sim.read(f) for f in FIELDS}, sim.adjoint(w[0], w[1])))
    for limit in (-1, 0):
        members = [make(**c) for c in cases]
        batch = D.Batch([m[0] for m in members])
        batch.set_block_steps(24)
        members[0][0].set_tape_limit(limit)
        for again in range(2):
            if again:
                for _, start, _ in members:
                    start()
            batch.record(steps, K)
            for (sim, _, _), (state, _) in zip(members, refs):
                for f in FIELDS:
                    assert np.array_equal(sim.read(f), state[f], equal_nan=True), (limit, again, f)
            got = batch.adjoint([m[2][0] for m in members], [m[2][1] for m in members])
            for g, (_, r) in zip(got, refs):
                for k in r:
                    assert np.array_equal(g[k], r[k]), (limit, again, k)
        batch.close()


# 20 x 34 listed tiles: the particle passes of the reverse steps go by tile,
# where the small mesh's go by particle (the mesh around the block does not
# enter its particles' results)
@pytest.mark.parametrize("name", list(CASES))
def test_reverse_by_tile_equals_by_particle(built, name):
    got = []
    for nx, ny in ((70, 50), (600, 500)):
        case = dict(CASES[name], nx=nx, ny=ny, split=1 << 30)
        if case.pop("loads", False):
            case.update(newtonian=True)     # (node ids differ between the meshes)
        sim, _, w = make(**case)
        sim.record(45, 45)
        got.append({**{f: sim.read(f) for f in FIELDS[:6]}, **sim.adjoint(w[0], w[1])})
    for k in got[0]:
        assert np.array_equal(got[0][k], got[1][k]), k
