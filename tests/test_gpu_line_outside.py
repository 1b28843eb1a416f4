"""A 1-D particle outside the mesh, at the start or after steps, is the out-of-mesh
error, for bars in one CTA and in separate kernels, with the per-step volume
set-up and the one at the start; the simulation can be set up again afterwards."""
import numpy as np
import pytest

import diffmpm_gb300 as D
from diffmpm_gb300._lib import OutOfMeshError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["usf", "usl"])
@pytest.mark.parametrize("reinit", [True, False])
@pytest.mark.parametrize("n", [1, 5, 2500])
def test_particle_outside(built, n, reinit, scheme):
    nx = max(4, n + 2)
    sim = D.Simulation(nx, 1.0, 1e-3, scheme=scheme, reinit_each_step=reinit, gravity=(0.0, 0.0), ndim=1,
                       materials=[D.LinearElastic({"density": 1.0, "youngs_modulus": 10.0, "poisson_ratio": 0.0})])
    inside = (np.arange(n) + 1.5).astype(np.float32).reshape(-1, 1)

    def start(loc, speed):
        sim.set_particles(loc, np.zeros(n, np.int32))
        sim.write("velocity", np.full(n, speed, np.float32))
        sim.initialize()

    for where in (-0.25, nx + 0.5, np.nan):
        loc = inside.copy()
        loc[n // 2] = where
        with pytest.raises(OutOfMeshError):
            start(loc, 0.0)
    start(inside, 50.0)                      # 0.05 elements a step, to the right
    with pytest.raises(OutOfMeshError):
        sim.step(60)
    start(inside, 50.0)
    sim.step(3)
    np.testing.assert_allclose(sim.read("loc"), inside[:, 0] + 0.15, rtol=1e-4)
