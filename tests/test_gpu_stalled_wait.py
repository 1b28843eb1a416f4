"""A wait between the CTAs of a resident sequence that runs out is an error the host
sees, and leaves the simulation where its step block began: the host's and the
device's step counters agree and the run goes on as if the call had not been
made.  The waits are made to give up at once (a limit of no reads at all)."""
import numpy as np
import pytest

from diffmpm_gb300._lib import MpmError
from test_gpu_resident import FIELDS, make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", [dict(), dict(scheme="usl", reinit=False, loads=True)], ids=["usf", "solve-usl-loads"])
@pytest.mark.parametrize("polls", [0, 1])
def test_wait_that_runs_out(built, polls, run):
    a, b = make("twenty-five", **run), make("twenty-five", **run)
    for sim in (a, b):
        sim.step(30)                          # blocks of 24 and 6 steps
    a.set_wait_polls(polls)
    before = {f: a.read(f) for f in FIELDS}
    with pytest.raises(MpmError, match="wait between the CTAs"):
        for _ in range(20):                   # (a wait may be over at its first read)
            a.step(24)
            b.step(24)
            before = {f: a.read(f) for f in FIELDS}
    assert a.step_index == b.step_index
    for f in FIELDS:
        assert np.array_equal(a.read(f), before[f]), f
    a.set_wait_polls(-1)
    for sim in (a, b):
        sim.step(40)
    assert a.step_index == b.step_index
    for f in FIELDS:
        assert np.array_equal(a.read(f), b.read(f)), f
    for f in ("mass", "velocity", "acceleration"):
        assert np.array_equal(a.read_nodal(f), b.read_nodal(f)), f
