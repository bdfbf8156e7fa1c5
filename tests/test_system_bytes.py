"""The footprint estimate of boxes with more cells than an int holds: rbmd_system_bytes runs before
rbmd_system_add looks at the description (the serving loop's admission), so it must answer, and the
system is refused when it is added."""
import os
import subprocess
import sys

import numpy as np
import pytest

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

SCRIPT = """
import sys
sys.path.insert(0, {root!r})
from tests.test_system_bytes import sparse
import rbmd_b200
print(rbmd_b200.system_bytes(sparse({edge})))
"""


def sparse(edge):
    """Two atoms in a box of edge^3 cells."""
    p = A.default_params(force_field=A.FF_LJ_CUT, neighbor=A.NEIGH_RBL, cut_off=1.0, r_core=1.0,
                         neighbor_sample_num=100, units=A.UNITS_LJ, timestep=0.001, temp_ctrl=A.TC_NONE)
    return synth.SystemData([[0.5] * 3, [2.5] * 3], np.ones(2), np.zeros(2), [1.0], [1.0], [0, 0, 0], [float(edge)] * 3,
                            params=p)


@pytest.mark.parametrize("edge", [1290, 2048, 65536, 10 ** 9])  # cells as an int: 2146689000, 0, 0, 0
def test_estimate_answers(edge):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=root, edge=edge)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
    assert int(r.stdout) > 2 ** 31


@pytest.mark.gpu
@pytest.mark.parametrize("edge", [1291, 2048, 65536])
def test_too_many_cells_are_refused(ctx_factory, edge):
    import rbmd_b200
    ctx = ctx_factory()
    with pytest.raises(rbmd_b200.RbmdError) as e:
        ctx.add_system(sparse(edge))
    assert e.value.code == A.ERR_UNSUPPORTED
    ctx.add_system(sparse(8))
