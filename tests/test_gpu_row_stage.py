"""The staged rows of the particle passes (RowStage16, csrc/mpm_device.cuh) where
the lanes of a warp part: rows of many chunks whose particles lie in drifted
and undrifted sort-cells, some past the row's cell map, with two materials.  The
reverse passes that stage rows give the bits of the ones that do not, and G2P by
whole tiles those of G2P by halves, for USF and USL (three and two chunks deep)."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

FIELDS = ("loc", "velocity", "stress", "strain", "density", "volumetric_strain_centroid")


def run(nx, ny, side, scheme):
    """22 x 14 cells of side x side jittered particles, every eleventh one fast
    enough to leave its cell within the run's single sort, in an nx x ny mesh."""
    rng = np.random.Generator(np.random.PCG64(side))
    h = 1.0 / 128
    mats = [D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e4, "poisson_ratio": 0.3}),
            D.Newtonian({"density": 900.0, "bulk_modulus": 1e4, "dynamic_viscosity": 1e-2})]
    sim = D.Simulation((nx, ny), (h, h), 2e-5, scheme=scheme, gravity=(0.5, -9.81), materials=mats)
    sim.set_empty_split(1 << 30)            # every tile is listed
    i, j = np.meshgrid(np.arange(8, 30), np.arange(6, 20))
    off = (np.arange(side) + 0.5) / side
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    n = x.size
    loc = (np.stack([x, y], 1) + rng.uniform(-0.3 / side, 0.3 / side, (n, 2))) * h
    vel = np.stack([np.sin(40 * loc[:, 1]), 0.3 * np.cos(30 * loc[:, 0])], 1)
    vel[::11] += rng.uniform(-12.0, 12.0, vel[::11].shape)
    sim.set_particles(loc.astype(np.float32), (rng.permutation(n) % 3 == 0).astype(np.int32))
    sim.write("velocity", vel.astype(np.float32))
    sim.write("youngs_modulus", (1e4 * np.exp(rng.uniform(-0.5, 0.5, n))).astype(np.float32))
    sim.set_block_steps(16)
    sim.initialize()
    w = rng.standard_normal((2, n, 2)).astype(np.float32)
    sim.record(16, 16)
    out = {f: sim.read(f) for f in FIELDS}
    assert sim.counters()["rollbacks"] == 0
    out.update(sim.adjoint(w[0], w[1]))
    sim.close()
    return out


# 12 tiles: passes by particle, G2P by halves of a tile; 20 x 34 tiles: by tile
@pytest.mark.parametrize("scheme", ["usf", "usl"])
@pytest.mark.parametrize("side", [1, 2, 5])   # 1, 4 and 25 particles a cell: 1, 3 and 18 chunks a row
def test_diverging_rows(built, side, scheme):
    a, b = run(70, 50, side, scheme), run(600, 500, side, scheme)
    for k in a:
        assert np.isfinite(a[k]).all() and np.array_equal(a[k], b[k]), k
