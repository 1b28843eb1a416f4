"""Recordings of a batch's members made together and apart: a member of a batch
stays an ordinary simulation, so its own adjoint after Batch.record, and the
batch's adjoint after each member recorded alone, give the bits of the call that
matches the recording -- kept whole or as checkpoints, in a fresh batch, after an
earlier recording of other particles' tiles, and with a rolled-back member."""
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


@pytest.mark.parametrize("limit,K", [(-1, 40), (-1, 20), (0, 20)])
@pytest.mark.parametrize("before", [False, True])
def test_batch_after_members_record(built, limit, K, before):
    out, batch = members(CASES, limit)
    refs = references(CASES, K)
    if before:                               # a recording of other tiles
        for sim, start, _ in out:
            loc = sim.read("loc")
            sim.write("loc", loc + np.float32(100.0 / 128))
            sim.initialize()
        batch.record(STEPS, K)
        batched(batch, out)
        for _, start, _ in out:
            start()
    for sim, _, _ in out:
        sim.record(STEPS, K)
    equal(batched(batch, out), refs, "recorded apart")
    batch.record(STEPS, K)
    for _, start, _ in out:
        start()
    batch.record(STEPS, K)
    out[0][1]()
    out[0][0].record(STEPS, K)               # one member again, alone
    equal(batched(batch, out), refs, "one member recorded apart")
    batch.close()
