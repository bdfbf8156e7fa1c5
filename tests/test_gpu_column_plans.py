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
