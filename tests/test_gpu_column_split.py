"""The two forms of the column pair kernel: a system alone, few chunks of atoms, has eight warps share a
chunk; in a batch of many chunks a warp takes one by itself.  An atom's force is formed row by row in
either, so the forces must be the same bit for bit.  Sizes with empty, partly filled and several chunks
per column, boxes whose stencils repeat cells, shell strides that are powers of two and not, atoms
outside the box (stray walks), and more traversal rows than the split form takes."""
import numpy as np
import pytest

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


def _water(n, **kw):
    return synth.saline(n, seed=n, **kw)


def _lj(cells, **kw):
    sd = synth.lj_fcc(cells=cells, precision=A.PREC_MIXED, rho=0.8, **kw)
    rng = np.random.default_rng(cells)
    sd.pos = sd.pos + rng.normal(scale=0.05, size=sd.pos.shape)  # some atoms end up outside the box
    return sd


CASES = {
    "water_1000": lambda: (_water(1000), _water(80000)),
    "water_2999": lambda: (_water(2999), _water(80000)),
    "water_9000": lambda: (_water(9000), _water(80000)),
    "water_philox": lambda: (_water(1500, rbl_mode=A.RBL_PHILOX), _water(80000)),
    "water_every_shell": lambda: (_water(1500, neighbor_sample_num=4000), _water(80000)),
    "water_odd_stride": lambda: (_water(1500, neighbor_sample_num=300), _water(80000)),
    "lj_49_rows": lambda: (_lj(6), _lj(28)),
    "lj_25_rows": lambda: (_lj(4, r_core=1.25), _lj(28, r_core=1.25)),
    "lj_81_rows": lambda: (_lj(6, r_core=0.7), _lj(28, r_core=0.7)),
}


@pytest.mark.parametrize("case", list(CASES))
def test_alone_and_in_a_large_batch_are_identical(ctx_factory, monkeypatch, case):
    monkeypatch.setenv("RBMD_PAIR_LAYOUT", "column")
    small, large = CASES[case]()
    alone, mixed = ctx_factory(), ctx_factory()
    a = alone.add_system(small)
    b = [mixed.add_system(small), mixed.add_system(large)]
    alone.init(a)
    mixed.init(b)
    assert np.array_equal(alone.forces(a), mixed.forces(b[0]))
    alone.step(a, 3)
    mixed.step(b, 3)
    assert np.array_equal(alone.forces(a), mixed.forces(b[0]))
    for x, y in zip(alone.state(a), mixed.state(b[0])):
        assert np.array_equal(x, y)
