"""mpm_step waits for its stream, also when it has no steps to run."""
import pytest

import diffmpm_gb300 as D
from diffmpm_gb300 import workloads

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, 1])
def test_step_waits_for_its_stream(built, steps):
    solver, g, _ = workloads.differentiation(D, n=16, sim_steps=1)
    sim = solver.simulation(g)
    solver._upload(sim)
    sim.initialize()
    stream, done = torch.cuda.Stream(), torch.cuda.Event()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)        # some 50 ms of work ahead on the stream
        done.record()
    sim.step(steps, stream=stream.cuda_stream)
    assert done.query()
