"""Field transfers and re-sorts of one simulation and of many in one launch
(csrc/mpm_sort.cu): every component comes back in original order, the
components no step touches included, and members re-sorted together end where
they end re-sorted alone."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu


def make(nx, ny, n, seed, reinit=True, speed=0.0):
    rng = np.random.Generator(np.random.PCG64(seed))
    h = 1.0 / 512
    mats = [D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3}),
            D.Newtonian({"density": 900.0, "bulk_modulus": 1e5, "dynamic_viscosity": 1e-3})]
    sim = D.Simulation((nx, ny), (h, h), 2e-5, reinit_each_step=reinit, gravity=(0.0, -9.81), materials=mats)
    lo, hi = 1.2 * h, np.array([nx - 1.2, ny - 1.2]) * h
    loc = rng.uniform(lo, np.minimum(hi, lo + 40 * h), size=(n, 2)).astype(np.float32)
    sim.set_particles(loc, rng.integers(0, 2, n).astype(np.int32))
    sim.write("velocity", (speed * np.sign(np.array([nx, ny]) * h / 2 - loc)).astype(np.float32))
    sim.initialize()
    return sim, loc


@pytest.mark.parametrize("n", [1, 255, 1025, 4099])
def test_every_component_comes_back(built, n):
    import torch
    sim, loc = make(45, 37, n, n, speed=3.0)
    rng = np.random.Generator(np.random.PCG64(7))
    stress = rng.standard_normal((n, 6)).astype(np.float32)
    strain = rng.standard_normal((n, 6)).astype(np.float32)
    sim.write("stress", stress)
    sim.write("strain", torch.from_numpy(np.concatenate([np.zeros(1, np.float32), strain.reshape(-1)]))
              .cuda()[1:])                                  # a device array four bytes off a 16-byte boundary
    assert np.array_equal(sim.read("stress"), stress) and np.array_equal(sim.read("strain"), strain)
    sim.write("stress", np.zeros((n, 6), np.float32) + stress * [0, 0, 0, 0, 1, 1])
    sim.step(3)
    assert np.array_equal(sim.read("stress")[:, 4:], stress[:, 4:])
    out = torch.empty(6 * n + 1, device="cuda")[1:]
    sim.read("strain", out=out)
    assert np.array_equal(out.view(n, 6)[:, [2, 4, 5]].cpu().numpy(), strain[:, [2, 4, 5]])
    assert np.array_equal(out.view(n, 6).cpu().numpy(), sim.read("strain"))


# one member of more than 2^18 cells (re-sorted by the kernels of a single
# simulation), uneven others; `fast` members drift in every block
@pytest.mark.parametrize("reinit", [True, False])
@pytest.mark.parametrize("shapes", [[(30, 20, 1), (64, 33, 2000), (91, 15, 777)],
                                    [(513, 513, 3000), (40, 40, 1024), (33, 70, 2500)], [(50, 31, 1500)]])
def test_members_resort_together_as_alone(built, shapes, reinit):
    alone = [make(nx, ny, n, 5 + k, reinit, speed=3.0)[0] for k, (nx, ny, n) in enumerate(shapes)]
    many = [make(nx, ny, n, 5 + k, reinit, speed=3.0) for k, (nx, ny, n) in enumerate(shapes)]
    batch = D.Batch([m[0] for m in many])
    fields = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid")
    start = {f: [s.read(f) for s in alone] for f in fields}
    for rounds in range(2):
        for f in fields:
            batch.write(f, np.concatenate([v.reshape(-1) for v in start[f]]))
        batch.write_nodal("velocity", np.zeros(sum(2 * s.nnodes for s in batch.sims), np.float32))
        batch.restart()
        batch.set_block_steps(20)
        batch.step(60)
        for k, s in enumerate(alone):
            for f in fields:
                s.write(f, start[f][k])
            s.write_nodal("velocity", np.zeros((s.nnodes, 2), np.float32))
            s.step_index = 0
            s.initialize()
            s.set_block_steps(20)
            s.step(60)
        for f in fields:
            got = batch.split(f, batch.read(f))
            for k, s in enumerate(alone):
                assert np.array_equal(got[k], s.read(f)), (f, k, rounds)
    assert sum(s.counters()["resorts"] for s in batch.sims) > 2 * len(shapes)
