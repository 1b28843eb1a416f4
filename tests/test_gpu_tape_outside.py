"""A particle that leaves the mesh in a recorded run is reported as in a plain run: the
steps after it read its position from the tape as the last step left it, not
what an earlier recording had there (which looked like a two-cell drift and had
the block replayed before the error)."""
import numpy as np
import pytest

import diffmpm_gb300 as D
from diffmpm_gb300._lib import OutOfMeshError

pytestmark = pytest.mark.gpu

NX, H, DT, STEPS = 64, 1.0 / 64, 1e-4, 24


@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("scheme", ["usf", "usl"])
def test_out_of_mesh_while_recording(built, scheme, batched):
    def simulation():
        return D.Simulation((NX, NX), (H, H), DT, scheme=scheme, gravity=(0.0, 0.0),
                            materials=[D.LinearElastic({"density": 1e3, "youngs_modulus": 1e3, "poisson_ratio": 0.3})])

    i, j = np.meshgrid(np.arange(50, NX), np.arange(10, 40))
    off = np.array([0.25, 0.75])
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    loc = (np.stack([x, y], 1) * H).astype(np.float32)

    def start(sim, loc, speed):
        sim.set_particles(loc, np.zeros(len(loc), np.int32))
        sim.write("velocity", np.tile(np.array([[speed, 0.0]], np.float32), (len(loc), 1)))
        sim.set_block_steps(STEPS)
        sim.initialize()

    sim = simulation()
    start(sim, loc[::-1] - np.array([[20 * H, 0]], np.float32), 0.0)   # elsewhere, in another order
    run = D.Batch([sim]) if batched else sim
    run.set_block_steps(STEPS)
    run.record(STEPS, STEPS)
    before = sim.counters()["rollbacks"]
    start(sim, loc, 0.8 * H / (STEPS * DT))               # the last column leaves after a third of the run
    with pytest.raises(OutOfMeshError):
        run.record(STEPS, STEPS)
    assert sim.counters()["rollbacks"] == before
