"""G2P by halves of a tile (fewer than 304 listed tiles) leaves what G2P by whole
tiles leaves, bit for bit: a simulation alone against a batch of one, whose
kernels take whole tiles, on meshes whose last tile row ends in the first half,
at the halves' border and in the second half, and on both sides of the limit;
drifting, with and without re-sorts."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

# node rows 5, 8, 9, 15, 16 + 8 of tiles of 31 x 15 nodes; 303 and 304 tiles
MESHES = [(40, 4), (33, 7), (33, 8), (70, 14), (70, 23), (92, 1514), (247, 569)]
FIELDS = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid", "volume", "mass")


def make(nx, ny, scheme, reinit, speed):
    rng = np.random.Generator(np.random.PCG64(nx + ny))
    h = 1.0 / 128
    sim = D.Simulation((nx, ny), (h, h), 4e-5, scheme=scheme, reinit_each_step=reinit, gravity=(0.0, -9.81),
                       materials=[D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3})])
    sim.set_empty_split(1 << 30)                     # every tile listed
    # blocks of 4 particles a cell: the mesh's middle, or its ends and middle
    rows = np.arange(1, ny - 1) if ny < 100 else np.r_[1:30, ny // 2 - 20:ny // 2 + 20, ny - 31:ny - 1]
    i, j, a, b = np.meshgrid(np.arange(1, nx - 1), rows, [0.25, 0.75], [0.25, 0.75], indexing="ij")
    loc = (np.stack([i + a, j + b], -1).reshape(-1, 2) + rng.uniform(-0.05, 0.05, (i.size, 2))) * h
    centre = np.array([nx, ny]) * h / 2
    sim.set_particles(loc.astype(np.float32))
    sim.write("velocity", (speed * (centre - loc) / (2 * centre)).astype(np.float32))   # inwards: stays in the mesh
    sim.set_block_steps(10)
    sim.initialize()
    return sim


@pytest.mark.parametrize("scheme,reinit,speed", [("usf", True, 10.0), ("usl", True, 10.0), ("usl", False, 10.0),
                                                 ("usf", False, 0.1)])
@pytest.mark.parametrize("nx,ny", MESHES)
def test_halves_equal_whole_tiles(built, nx, ny, scheme, reinit, speed):
    alone, member = make(nx, ny, scheme, reinit, speed), make(nx, ny, scheme, reinit, speed)
    batch = D.Batch([member])
    batch.set_block_steps(10)
    for _ in range(5):                               # (5 steps a call: one launch a phase)
        alone.step(5)
        batch.step(5)
    for f in FIELDS:
        assert np.array_equal(alone.read(f), member.read(f)), f
    for f in ("mass", "velocity", "acceleration"):
        assert np.array_equal(alone.read_nodal(f), member.read_nodal(f)), f
