"""RBE sampling at the edges of its rounds of proposal slots: one sample, counts around a word and
around a round, many rounds, distributions that are mostly the zero vector (more slots than samples),
and one that never leaves it (the slot limit).  Integer work: equal to the oracle's."""
import numpy as np
import pytest

from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha", [0.6, 0.02, 0.004])
@pytest.mark.parametrize("P", [1, 2, 33, 959, 960, 961, 1024, 2100, 8192])
def test_samples_match_oracle(ctx_factory, oracle_mod, P, alpha):
    sd = synth.nacl_melt(n_side=8, P=P, alpha=alpha, seed=P + 3)
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.compute_forces(sid)
    o = oracle_mod.Oracle(sd)
    o.compute_forces()
    assert np.array_equal(ctx.kspace(sid)[0], o.kspace()[0])


def test_slot_limit_matches_oracle(ctx_factory, oracle_mod):
    sd = synth.nacl_melt(n_side=8, P=5, alpha=1e-6)
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.compute_forces(sid)
    o = oracle_mod.Oracle(sd)
    o.compute_forces()
    assert np.array_equal(ctx.kspace(sid)[0], o.kspace()[0])
    assert ctx.thermo(sid)["status"] & 32
