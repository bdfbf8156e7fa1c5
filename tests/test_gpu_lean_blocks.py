"""The lean pair kernel's two register budgets (FP64, special bonds): a system alone whose blocks fill the
chip once or twice takes the one of two blocks per SM (up to 2368 atoms, and 3553 to 4736, on 148 SMs), in
a batch of many atoms the other.  The same arithmetic in the same order: forces and trajectories must be
the same bit for bit, on both sides of each line."""
import numpy as np
import pytest

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [{}, {"neighbor": A.NEIGH_VERLET, "coulomb": A.COUL_EWALD}], ids=["rbl_rbe", "verlet_ewald"])
@pytest.mark.parametrize("n_mol", [340, 789, 790, 1184, 1185, 1578, 1579, 2729])
def test_few_and_many_atoms_are_identical(ctx_factory, kw, n_mol):
    small = synth.spce_water(n_mol=n_mol, seed=3, precision=A.PREC_FP64, **kw)
    large = synth.spce_water(n_mol=3000, seed=4, precision=A.PREC_FP64, **kw)
    alone, mixed = ctx_factory(), ctx_factory()
    a = alone.add_system(small)
    b = [mixed.add_system(small), mixed.add_system(large)]
    alone.init(a)
    mixed.init(b)
    assert np.array_equal(alone.forces(a), mixed.forces(b[0]))
    alone.step(a, 2)
    mixed.step(b, 2)
    for x, y in zip(alone.state(a), mixed.state(b[0])):
        assert np.array_equal(x, y)
