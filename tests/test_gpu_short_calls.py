"""A call of a few steps costs no more than one of a few more (loops of short calls,
as solve and outputs every few steps make them): 7 steps against 8, where a launch
a phase once took twice the time of the 8 in one launch."""
import time

import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["usf", "usl"])
@pytest.mark.parametrize("nx", [10, 118])      # one tile and a part of a wave
def test_seven_steps_cost_less_than_eight(built, nx, scheme):
    sim = D.Simulation((nx, nx), (1.0 / nx, 1.0 / nx), 1e-5 / nx, scheme=scheme, gravity=(0.0, -9.81),
                       materials=[D.LinearElastic({"density": 1e3, "youngs_modulus": 1e5, "poisson_ratio": 0.3})])
    i, j = np.meshgrid(np.arange(nx // 8, nx - nx // 8), np.arange(0, nx // 2))
    off = np.array([0.25, 0.75])
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    sim.set_particles((np.stack([x, y], 1) / nx).astype(np.float32))
    sim.initialize()

    def call(m):
        t0 = time.perf_counter()
        for _ in range(20):
            sim.step(m)
        return time.perf_counter() - t0

    t = np.min([[call(7), call(8)] for _ in range(12)], axis=0)
    assert t[0] < 1.1 * t[1], t / 20
