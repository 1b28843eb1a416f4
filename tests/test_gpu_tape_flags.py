"""The drift flags of a taped segment belong to that segment: a recording of a body
at rest takes the fast path in every step, also on a handle whose earlier
recording left flags where now no particle is (such a tile is not among the
steps' tiles, so no step writes its flags).  The results do not depend on it, so
the times of the two recordings are compared."""
import time

import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

STEPS = 40
NX, NY, H, DT = 70, 2000, 1.0 / 128, 2e-5


def block(i0, i1):
    i, j = np.meshgrid(np.arange(i0, i1), np.arange(4, NY - 4))
    off = (np.arange(4) + 0.5) / 4
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    return (np.stack([x, y], 1) * H).astype(np.float32)


def simulation():
    sim = D.Simulation((NX, NY), (H, H), DT, gravity=(0.0, 0.0),
                       materials=[D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e4, "poisson_ratio": 0.3})])
    sim.set_empty_split(0)
    return sim


def start(sim, loc, speed):
    sim.set_particles(loc, np.zeros(len(loc), np.int32))
    sim.write("velocity", np.tile(np.array([[speed, 0.0]], np.float32), (len(loc), 1)))
    sim.set_block_steps(STEPS)
    sim.initialize()


def record(sim, seeds):
    t0 = time.perf_counter()
    sim.record(STEPS, STEPS)
    sim.adjoint(seeds)
    return time.perf_counter() - t0


def test_flags_of_an_earlier_recording(built):
    # tile columns own cells 0..30, 31..61, ...; those of the second see cells
    # from 29 on.  The first body moves about a cell across them.
    moving, still = block(10, 36), block(33, 59)
    seeds = np.ones_like(still)
    used, fresh = simulation(), simulation()
    start(used, moving, 1.0 * H / (STEPS * DT))
    record(used, seeds)
    for sim in (used, fresh):
        start(sim, still, 0.0)
    t = np.min([[record(used, seeds), record(fresh, seeds)] for _ in range(15)], axis=0)
    print(f"recording and adjoint {1e3 * t[0]:.2f} ms, on a fresh handle {1e3 * t[1]:.2f}")
    # the same work; with the earlier flags every taped step gathers (1.28 times the time)
    assert t[0] < 1.12 * t[1]
