"""Batches whose members differ in what they hold -- a Newtonian material, particle
moduli, velocity constraints, nodal forces -- give every member the gradients that
it has alone, bit for bit."""
import numpy as np
import pytest

import diffmpm_gb300 as D
from test_gpu_tape import make

pytestmark = pytest.mark.gpu

STEPS, K = 30, 10
MEMBERS = [dict(newtonian=True, seed=4), dict(seed=5, nx=61, ny=47), dict(newtonian=True, seed=6, nx=44, ny=40),
           dict(seed=7, nx=90, ny=33, speed=8.0)]


def plain(spec, scheme, reinit, moduli):
    sim, start, w = make(scheme=scheme, reinit=reinit, **spec)
    if not moduli:                            # the materials' own moduli
        loc, vel = sim.read("loc"), sim.read("velocity")
        mid = sim.read("material_id")
        sim.set_particles(loc, mid)
        sim.write("velocity", vel)
        if spec["seed"] % 2:
            sim.set_particle_velocity_constraints([sim.n // 2, 3], [0, 1], [0.1, 0.0])
        sim.initialize()
    return sim, w


@pytest.mark.parametrize("reinit", [True, False])
@pytest.mark.parametrize("scheme", ["usf", "usl"])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (1, 0), (3, 1, 0)])
def test_members_with_and_without(built, order, scheme, reinit):
    specs = [MEMBERS[k] for k in order]
    refs = []
    for k, spec in enumerate(specs):
        sim, w = plain(spec, scheme, reinit, k % 2 == 0)
        sim.record(STEPS, K)
        refs.append(sim.adjoint(w[0], w[1]))
    members = [plain(spec, scheme, reinit, k % 2 == 0) for k, spec in enumerate(specs)]
    batch = D.Batch([m[0] for m in members])
    batch.set_block_steps(24)
    for sim, _ in members:
        sim.set_block_steps(24)
    batch.record(STEPS, K)
    got = batch.adjoint([w[0] for _, w in members], [w[1] for _, w in members])
    for g, r in zip(got, refs):
        for k in r:
            assert np.isfinite(r[k]).all() and np.array_equal(g[k], r[k]), k
    batch.close()
