"""The one-CTA 1-D step and reverse step (csrc/mpm_line.cu, mpm_line_adjoint.cu)
against the kernel-per-phase path, which longer meshes take.

A bar keeps its elements' length, particles and loads when empty elements are
added at its far end, and 2047 elements run in one CTA where 2048 run as
separate kernels: both must give the same bits, forward and reverse.  Sizes
straddle a warp, one and two particles a thread and the particle limit; the
fast bars change element in most steps."""
import numpy as np
import pytest

import diffmpm_gb300 as D

pytestmark = pytest.mark.gpu

H = 1.0 / 512


def run(nx, n, scheme, reinit, speed, steps=24):
    rng = np.random.Generator(np.random.PCG64(n))
    ppe = max(1, n // 400)
    x = ((np.arange(n) // ppe + 1) + (np.arange(n) % ppe + 0.5 + rng.uniform(-0.2, 0.2, n)) / ppe) * H
    order = rng.permutation(n)              # original order unrelated to position
    x = x[order]
    fn = D.Linear(0, np.array([0.0, 4e-5]), np.array([0.0, 1.0]))
    mats = [D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e6, "poisson_ratio": 0.3}),
            D.Newtonian({"density": 1000.0, "bulk_modulus": 1e6, "dynamic_viscosity": 5.0})]
    sim = D.Simulation(nx, H, 2e-6, scheme=scheme, reinit_each_step=reinit, gravity=(-9.81, 0.0), ndim=1,
                       constraints=[(np.array([0]), D.Constraint(0, 0.0))], functions=[fn],
                       nodal_forces=[D.NodalForce(np.array([2]), fn, 0, 0.5)], materials=mats)
    sim.set_particles(x.astype(np.float32), (np.arange(n) % 5 == 0).astype(np.int32))
    sim.write("velocity", (speed + 0.5 * np.sin(30 * x)).astype(np.float32))
    sim.write("youngs_modulus", (1e6 * rng.uniform(0.5, 2.0, n)).astype(np.float32))
    sim.set_particle_velocity_constraints(np.array([n // 2]), np.array([0]), np.array([speed]))
    sim.initialize()
    sim.step(7)                             # an odd count: the ping-pong parity changes
    sim.record(steps)
    out = {k: sim.read(k) for k in ("loc", "velocity", "stress", "strain", "density", "volume", "mass",
                                    "volumetric_strain_centroid", "element_ids")}
    for k in ("mass", "velocity", "acceleration"):
        out["nodal " + k] = sim.read_nodal(k)[: 2048 - 1]
    w = rng.standard_normal((2, n, 1)).astype(np.float32)
    out.update({"d " + k: v for k, v in sim.adjoint(w[0], w[1]).items()})
    return out


@pytest.mark.parametrize("speed", [0.5, 400.0])
@pytest.mark.parametrize("n,scheme,reinit", [(1, "usl", True), (32, "usf", True), (33, "usl", False),
                                             (1024, "usf", False), (1025, "usl", True), (2048, "usf", True)])
def test_one_cta_equals_kernel_per_phase(built, n, scheme, reinit, speed):
    a, b = (run(nx, n, scheme, reinit, speed) for nx in (2047, 2048))
    for k in a:
        assert np.isfinite(a[k]).all(), k
        assert np.array_equal(a[k], b[k]), k


def test_particle_limit(built):
    """One particle more than a CTA takes runs as separate kernels: its
    neighbours' results do not depend on which path that is."""
    a, b = run(2047, 2049, "usf", True, 0.5), run(2048, 2049, "usf", True, 0.5)
    for k in a:
        assert np.array_equal(a[k], b[k]), k
