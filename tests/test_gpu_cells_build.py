"""Cell lists where the build kernel's branches part: cells with more atoms than a bucket holds (the
overflow list), boxes of more cells than are added up in one level, boxes of a few cells, and lists
built one after the other from the two count buffers.  Integer work: equal to the oracle's."""
import numpy as np
import pytest

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


def _lj(n, box, pos):
    p = A.default_params(force_field=A.FF_LJ_CUT, neighbor=A.NEIGH_RBL, cut_off=2.5, r_core=1.2,
                         neighbor_sample_num=100, units=A.UNITS_LJ, timestep=0.005, temp_ctrl=A.TC_NONE)
    return synth.SystemData(pos, np.ones(n), np.zeros(n), [1.0], [1.0], [0, 0, 0], [box] * 3, params=p)


def _positions(kind, n, box, rng):
    if kind == "spread":
        return rng.uniform(0, box, (n, 3))
    if kind == "one_cell":  # every atom in the last cell
        return box - rng.uniform(0, 0.5, (n, 3))
    k = n // 2  # two crowded cells among an empty box, and atoms outside it
    pos = rng.uniform(0, box, (n, 3))
    pos[:k] = 0.3 + rng.uniform(0, 0.2, (k, 3))
    pos[k:k + 20] = box + rng.uniform(0, 0.3, (20, 3))
    return pos


@pytest.mark.parametrize("kind", ["spread", "one_cell", "crowded"])
@pytest.mark.parametrize("n,box", [(40, 7.6), (700, 9.0), (3000, 16.0), (900, 27.0)])
def test_cells_match_oracle(ctx_factory, oracle_mod, kind, n, box):
    rng = np.random.default_rng(n)
    ctx = ctx_factory()
    sd = _lj(n, box, _positions(kind, n, box, rng))
    sid = ctx.add_system(sd)
    for turn in range(3):
        if turn:
            sd = _lj(n, box, _positions(kind if turn == 2 else "spread", n, box, rng))
            ctx.set_state(sid, x=sd.pos)
        for a, b in zip(ctx.cells(sid), oracle_mod.Oracle(sd).cells()):
            assert np.array_equal(a, b)
