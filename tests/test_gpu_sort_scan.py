"""The scan of a re-sort's cell counts in one launch (up to 2^18 cells) and in
three (above): the storage order after it is that of a stable sort by cell, for
meshes of less than a piece, around whole chunks of 16384 counts and on both
sides of the limit, alone and in a batch."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

# cells: 3, 4, 16383 to 16385 (chunk edges count one entry more), 2^18, 2^18 + 512
MESHES = [(3, 1), (2, 2), (127, 129), (128, 128), (113, 145), (512, 512), (512, 513), (301, 407)]


def make(nx, ny, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    h = 1.0 / 64
    n = 4000
    sim = D.Simulation((nx, ny), (h, h), 1e-5, materials=[
        D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3})])
    loc = (rng.uniform(0.0, 1.0, (n, 2)) * [nx, ny]).astype(np.float32)
    loc[:3] = [[0.25, 0.25], [nx - 0.5, ny - 0.5], [nx - 0.5, 0.5]]
    loc = (np.minimum(loc, np.float32([nx, ny]) * np.float32(0.9999)) * np.float32(h)).astype(np.float32)
    sim.set_particles(loc)
    return sim, loc


def check(sim, loc, nx):
    h = np.float32(1.0 / 64)                                   # a power of two: exact cells
    cell = (loc[:, 1] // h).astype(np.int64) * nx + (loc[:, 0] // h).astype(np.int64)
    assert np.array_equal(sim.read("element_ids").reshape(-1), cell)
    held = np.rint(float(h) ** 2 / sim.read("volume").reshape(-1).astype(np.float64))   # a cell's volume / its count
    assert np.array_equal(held.astype(np.int64), np.bincount(cell)[cell])


@pytest.mark.parametrize("nx,ny", MESHES)
def test_scan_sizes(built, nx, ny):
    sim, loc = make(nx, ny, nx)
    sim.initialize()
    check(sim, loc, nx)
    sim.step(1)                                                # (the order the kernels use)
    assert np.isclose(sim.read_nodal("mass").sum(dtype=np.float64),
                      np.unique((loc // np.float32(1.0 / 64)).astype(int), axis=0).shape[0] * 1000.0 / 64 ** 2,
                      rtol=1e-5)


def test_scan_of_many(built):
    sims = [make(nx, ny, nx) for nx, ny in MESHES]
    for s, _ in sims:
        s.initialize()
    batch = D.Batch([s for s, _ in sims])
    moved = [np.ascontiguousarray(loc[::-1]) for _, loc in sims]
    batch.write("loc", np.concatenate([m.reshape(-1) for m in moved]))
    batch.restart()
    for (s, _), loc, (nx, _) in zip(sims, moved, MESHES):
        check(s, loc, nx)
