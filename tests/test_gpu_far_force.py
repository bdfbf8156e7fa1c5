"""Structure factor and far force at the edges of their blocks: atom counts around 64, 128 and 256 (and
around the sizes where the structure factor's blocks grow), k counts around a lane group and a staged
tile, every warp's share of a chunk empty or partly filled.

The structure factor is compared with a direct sum: FP64 to n times the rounding of a phase of a few
hundred (1e-13 each); mixed precision to 1e-6 per term, the SFU sine's error on a phase reduced in FP32.
Forces are compared with the oracle at the tolerances of the force parity tests."""
import numpy as np
import pytest

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

from conftest import rel_rms

pytestmark = pytest.mark.gpu


def _ions(n, P, precision):
    """n ions on random sites of a cubic lattice, spacing 1.2, neutral or one charge off."""
    side = max(6, int(np.ceil(n ** (1 / 3) - 1e-9)))
    rng = np.random.default_rng(n + P)
    sites = np.sort(rng.choice(side ** 3, n, replace=False))
    pos = np.stack(np.unravel_index(sites, (side,) * 3), -1) * 1.2 + 0.6 + rng.normal(scale=0.05, size=(n, 3))
    base = synth.nacl_melt(n_side=8, P=P, precision=precision, seed=P)
    return synth.SystemData(pos, np.ones(n), (np.arange(n) % 2).astype(np.int32), base.eps, base.sig, [0, 0, 0],
                            [1.2 * side] * 3, charge=np.where(np.arange(n) % 2 == 0, 1.0, -1.0), params=base.params)


@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_MIXED])
@pytest.mark.parametrize("n,P", [(8, 1), (63, 31), (64, 32), (65, 33), (200, 257), (256, 256), (257, 100), (1000, 511),
                                 (9472, 40), (9473, 40), (18944, 9), (18945, 9)])
def test_structure_factor_is_the_direct_sum(ctx_factory, n, P, precision):
    sd = _ions(n, P, precision)
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.compute_forces(sid)
    m, rho = ctx.kspace(sid)
    ph = sd.pos @ (2 * np.pi * m / sd.box_hi).T
    want = np.stack([sd.charge @ np.cos(ph), sd.charge @ np.sin(ph)], -1)
    per_atom = 1e-13 if precision == A.PREC_FP64 else 1e-6
    assert np.abs(rho - want).max() < n * per_atom


@pytest.mark.parametrize("precision,tol", [(A.PREC_FP64, 1e-9), (A.PREC_MIXED, 1e-4)])
@pytest.mark.parametrize("n,P", [(63, 31), (64, 32), (65, 3), (256, 257), (257, 100), (1000, 511)])
def test_forces_match_oracle(ctx_factory, oracle_mod, n, P, precision, tol):
    sd = _ions(n, P, precision)
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.compute_forces(sid)
    o = oracle_mod.Oracle(sd)
    o.compute_forces()
    assert rel_rms(ctx.forces(sid), o.forces()) < tol


@pytest.mark.parametrize("kind,P", [("water", 100), ("water", 300), ("ions", 200)])
def test_assembly_of_a_large_batch_forms_the_same_forces(ctx_factory, kind, P):
    """In batches of two million atoms and more the force assembly forms the far force and the
    intramolecular terms itself.  The same sums in the same order: a small system alone and in such a
    batch must agree bit for bit, also with more k vectors than are staged at a time."""
    if kind == "water":
        small, fill, count = synth.saline(1300, seed=1, P=P), synth.saline(64000, seed=2, P=P), 32
    else:
        small = synth.nacl_melt(n_side=12, P=P, precision=A.PREC_MIXED, seed=1)
        fill, count = synth.nacl_melt(n_side=64, P=P, precision=A.PREC_MIXED, seed=2), 8
    alone, large = ctx_factory(), ctx_factory()
    a = alone.add_system(small)
    b = [large.add_system(small)] + [large.add_system(fill) for _ in range(count)]
    assert small.n + count * fill.n > 2000000
    alone.init(a)
    large.init(b)
    assert np.array_equal(alone.forces(a), large.forces(b[0]))
    alone.step(a, 2)
    large.step(b, 2)
    assert np.array_equal(alone.forces(a), large.forces(b[0]))
    for x, y in zip(alone.state(a), large.state(b[0])):
        assert np.array_equal(x, y)
