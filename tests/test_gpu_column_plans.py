"""Column-layout systems of different traversal row counts in one process.  Each kernel of the split form
takes dynamic shared memory by the batch's rows, and a limit on it belongs to the kernel, not to the
batch: a batch planned later, with fewer rows, must not lower what an earlier one launches with.  More
rows first, in one call and in turns, the forms with eight and with sixteen warps per chunk; forces equal
to those of each system in a context of its own, bit for bit."""
import numpy as np
import pytest

import rbmd_b200
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu

# eight warps per chunk: 49 and 25 rows; sixteen: 25 and 9 rows
PAIRS = {
    "eight_warps": lambda: (synth.saline(3000, seed=1, r_core=4.0), synth.saline(9000, seed=2)),
    "sixteen_warps": lambda: (synth.saline(1200, seed=1), synth.saline(1200, seed=2, r_core=10.0)),
}


@pytest.fixture(params=list(PAIRS))
def pair(request, monkeypatch):
    monkeypatch.setenv("RBMD_PAIR_LAYOUT", "column")
    return PAIRS[request.param]()


def _alone(ctx_factory, sd, steps):
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.init(sid)
    if steps:
        ctx.step(sid, steps)
    return ctx.forces(sid)


def test_a_step_that_cannot_be_captured_leaves_nothing_behind(ctx_factory, pair):
    """Where a step's launches cannot be captured it is an error each time, and the next call of another
    system does not report it again."""
    init, stepped = [_alone(ctx_factory, sd, 0) for sd in pair], [_alone(ctx_factory, sd, 2) for sd in pair]
    ctx = ctx_factory()
    ids = []
    for sd, f in zip(pair, init):  # one by one, each right after its own plan
        ids.append(ctx.add_system(sd))
        ctx.init(ids[-1])
        assert np.array_equal(ctx.forces(ids[-1]), f)
    done = 0
    for _ in range(2):
        try:
            ctx.step(ids, 1)
            done += 1
        except rbmd_b200.RbmdError:
            ctx.compute_forces(ids[1])
            assert np.array_equal(ctx.forces(ids[1]), init[1])
    assert done in (0, 2)
    if done:
        for sid, f in zip(ids, stepped):
            assert np.array_equal(ctx.forces(sid), f)


def test_forces_of_one_call_and_in_turns(ctx_factory, pair):
    init = [_alone(ctx_factory, sd, 0) for sd in pair]
    stepped = [_alone(ctx_factory, sd, 2) for sd in pair]
    ctx = ctx_factory()
    ids = [ctx.add_system(sd) for sd in pair]
    ctx.init(ids)
    for sid, f in zip(ids, init):
        assert np.array_equal(ctx.forces(sid), f)
    for turn in (0, 1, 0):  # positions unchanged: the same forces again
        ctx.compute_forces(ids[turn])
        assert np.array_equal(ctx.forces(ids[turn]), init[turn])
    ctx.step(ids, 2)
    for sid, f in zip(ids, stepped):
        assert np.array_equal(ctx.forces(sid), f)
    ctx.thermo(ids[0])


def test_a_second_context_does_not_disturb_the_first(ctx_factory, pair):
    init = _alone(ctx_factory, pair[0], 0)
    first, second = ctx_factory(), ctx_factory()
    a = first.add_system(pair[0])
    first.init(a)
    b = second.add_system(pair[1])
    second.init(b)
    first.compute_forces(a)
    assert np.array_equal(first.forces(a), init)
