"""A member of a batch stays an ordinary simulation: its own adjoint after
Batch.record gives the bits of a recording of its own -- kept whole or as
checkpoints, and with a rolled-back member."""
import numpy as np
import pytest

import diffmpm_gb300 as D
from test_gpu_tape import make

pytestmark = pytest.mark.gpu

STEPS = 40
CASES = [dict(nx=220, ny=130, seed=5), dict(nx=170, ny=150, seed=6, velocity_update=True)]
THROWN = dict(nx=220, ny=130, seed=7, speed=40.0)


def members(cases, limit):
    out = [make(**c) for c in cases]
    for sim, _, _ in out:
        sim.set_tape_limit(limit)
    batch = D.Batch([m[0] for m in out])
    batch.set_block_steps(24)
    return out, batch


def gradients(sim, w):
    return sim.adjoint(w[0], w[1])


def references(cases, K):
    refs = []
    for c in cases:
        sim, _, w = make(**c)
        sim.record(STEPS, K)
        refs.append(gradients(sim, w))
    return refs


def equal(got, refs, why):
    for i, (g, r) in enumerate(zip(got, refs)):
        for k in r:
            assert np.isfinite(r[k]).all() and np.array_equal(g[k], r[k]), (why, i, k)


def batched(batch, out):
    return batch.adjoint([m[2][0] for m in out], [m[2][1] for m in out])


@pytest.mark.parametrize("limit,K", [(-1, 40), (-1, 20), (0, 20)])
@pytest.mark.parametrize("thrown", [False, True])
def test_member_after_batch_record(built, limit, K, thrown):
    cases = CASES + [THROWN] if thrown else CASES
    out, batch = members(cases, limit)
    refs = references(cases, K)
    batch.record(STEPS, K)
    equal([gradients(m[0], m[2]) for m in out], refs, "each member")
    equal(batched(batch, out), refs, "the batch after its members")
    equal([gradients(m[0], m[2]) for m in out], refs, "each member again")
    if thrown:
        assert out[-1][0].counters()["rollbacks"] > 0
    batch.close()
