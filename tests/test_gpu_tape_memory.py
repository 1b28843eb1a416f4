"""The device memory that recordings hold: no more than a bounded multiple of what
their checkpoint interval asks for unless the caller sets another bound, and
given back when a later recording may keep or needs less -- for one simulation, a
batch, the autograd function and a bar; the gradients are the same bits."""
import gc

import numpy as np
import pytest

import diffmpm_gb300 as D
from diffmpm_gb300 import workloads
from diffmpm_gb300.autograd import explicit_run

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 256                 # mesh side; 160 x 160 cells of 4 particles
NP = 160 * 160 * 4
# bytes of a taped step and of a checkpoint, by their arrays: 9 floats a
# particle, 7 a node and a flag a cell; 14 words and a byte a particle, two
# floats a node, a word and a byte a cell
SLOT = NP * 36 + (N + 1) ** 2 * 28 + N * N
CHECKPOINT = NP * 57 + (N + 1) ** 2 * 8 + N * N * 5


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def simulation():
    h = 1.0 / N
    sim = D.Simulation((N, N), (h, h), 1e-5, gravity=(0.0, -9.81),
                       materials=[D.LinearElastic({"density": 1000.0, "youngs_modulus": 1e5, "poisson_ratio": 0.3})])
    i, j = np.meshgrid(np.arange(40, 200), np.arange(20, 180))
    off = np.array([0.25, 0.75])
    x = (i[..., None, None] + off + 0 * off[:, None]).reshape(-1)
    y = (j[..., None, None] + 0 * off + off[:, None]).reshape(-1)
    loc = (np.stack([x, y], 1) * h).astype(np.float32)

    def start():
        sim.set_particles(loc, np.zeros(NP, np.int32))
        sim.initialize()

    start()
    return sim, start


def recorded(sim, start, steps, K):
    start()
    sim.record(steps, K)
    held = used()
    return held, sim.adjoint(np.ones((NP, 2), np.float32))


def test_lowered_bound_and_shorter_run_give_back(built):
    sim, start = simulation()
    start()
    base = used()
    whole, g0 = recorded(sim, start, 120, 40)       # whole: three times the segment
    assert whole - base > 120 * SLOT
    sim.set_tape_limit(0)
    kept, g1 = recorded(sim, start, 120, 40)        # a segment and four checkpoints
    assert kept < whole - 40 * SLOT
    for k in g0:
        assert np.array_equal(g0[k], g1[k]), k
    sim.set_tape_limit(-1)
    whole, _ = recorded(sim, start, 120, 40)
    short, _ = recorded(sim, start, 8, 8)
    assert short < whole - 100 * SLOT


def test_interval_bounds_the_tape(built):
    sim, start = simulation()
    start()
    base = used()
    steps, K = 400, 10
    asked = 41 * CHECKPOINT + K * SLOT
    held, g0 = recorded(sim, start, steps, K)
    # (a sort epoch, adjoint buffers and copy tables come on top)
    assert held - base < 2 * asked
    sim.set_tape_limit(1 << 33)                     # the caller's own bound
    whole, g1 = recorded(sim, start, steps, K)
    assert whole - base > steps * SLOT
    for k in g0:
        assert np.array_equal(g0[k], g1[k]), k


def test_batch_and_autograd_bounds(built):
    pairs = [simulation() for _ in range(2)]
    batch = D.Batch([p[0] for p in pairs])
    batch.record(120, 40)
    whole = used()
    batch.set_tape_limit(0)
    for _, start in pairs:
        start()
    batch.record(120, 40)
    assert used() < whole - 2 * 40 * SLOT
    batch.close()
    for sim, _ in pairs:
        sim.close()

    solver, g, info = workloads.differentiation(D, n=N, sim_steps=120)
    dev = torch.device("cuda:0")
    grads, held = [], []
    for limit in (-1, 0, -1):
        gc.collect()
        E = torch.full((info["np"],), 1e6, device=dev, requires_grad=True)
        x, v = explicit_run(solver, g, E, checkpoint_steps=40, tape_limit=limit)
        held.append(used())
        x.square().sum().backward()
        grads.append(E.grad.clone())
        del x, v
    assert held[1] < held[0] - 40 * SLOT
    assert torch.equal(grads[0], grads[1]) and torch.equal(grads[0], grads[2])


def test_bar_gives_back(built):
    sim = D.Simulation((2000,), (1.0,), 1e-3, ndim=1, gravity=(0.0, 0.0),
                       materials=[D.LinearElastic({"density": 1.0, "youngs_modulus": 100.0, "poisson_ratio": 0.0})])
    loc = (np.arange(2000) + 0.5).astype(np.float32).reshape(-1, 1)

    def record(steps):
        sim.set_particles(loc, np.zeros(len(loc), np.int32))
        sim.initialize()
        sim.record(steps)
        return used()

    long = record(2000)
    assert record(10) < long - 2000 * 2000 * 40 // 2
