"""Momentum of 1-D particles, read before anything re-sorts them: the mass counts the
particles that an element held at the start of the last step, the same whether
the steps ran in one CTA (2047 elements) or as separate kernels (2048)."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

H = 1.0 / 512


@pytest.mark.parametrize("reinit", [True, False])
@pytest.mark.parametrize("scheme", ["usf", "usl"])
def test_momentum_after_steps(built, scheme, reinit):
    rng = np.random.Generator(np.random.PCG64(8))
    n = 700
    x = ((np.arange(n) // 3 + 1) + (np.arange(n) % 3 + 0.5 + rng.uniform(-0.2, 0.2, n)) / 3)[rng.permutation(n)] * H
    out = []
    for nx in (2047, 2048):
        sim = D.Simulation(nx, H, 2e-6, scheme=scheme, reinit_each_step=reinit, gravity=(-9.81, 0.0), ndim=1,
                           materials=[D.LinearElastic({"density": 1e3, "youngs_modulus": 1e6, "poisson_ratio": 0.3})])
        sim.set_particles(x.astype(np.float32), np.zeros(n, np.int32))
        sim.write("velocity", (300.0 + 200.0 * np.sin(30 * x)).astype(np.float32))
        sim.initialize()
        got = []
        for steps in (1, 7, 16):
            sim.step(steps)
            got.append(sim.read("momentum"))
        sim.record(9)
        got.append(sim.read("momentum"))
        out.append(got + [sim.read("volume"), sim.read("momentum")])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.isfinite(a).all() and np.array_equal(a, b), k
