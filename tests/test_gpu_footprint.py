"""Device memory that adding a system takes: one allocation of about the estimated footprint.  A force
field without charges has no k-space arrays, whatever its Coulomb method is set to."""
import numpy as np
import pytest
import torch

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


def _taken(ctx_factory, coulomb):
    n_side = 160
    g = np.arange(n_side) * 1.2 + 0.6
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    p = A.default_params(force_field=A.FF_LJ_CUT, neighbor=A.NEIGH_RBL, cut_off=2.4, r_core=2.4, coulomb=coulomb,
                         coulomb_sample_num=100, alpha=0.1, kmax=(3, 3, 3), neighbor_sample_num=100, units=A.UNITS_LJ,
                         timestep=0.001, temp_ctrl=A.TC_NONE)
    sd = synth.SystemData(pos, np.ones(len(pos)), np.zeros(len(pos)), [1.0], [1.0], [0, 0, 0], [1.2 * n_side] * 3,
                          params=p)
    ctx = ctx_factory()
    small = ctx.add_system(synth.lj_fcc(cells=4))
    ctx.state(small)
    before = torch.cuda.mem_get_info()[0]
    ctx.add_system(sd)
    return before - torch.cuda.mem_get_info()[0], len(pos)


def test_no_k_space_memory_without_charges(ctx_factory):
    torch.cuda.init()
    plain, n = _taken(ctx_factory, A.COUL_NONE)
    rbe, _ = _taken(ctx_factory, A.COUL_RBE)
    assert plain > 200 * n
    assert rbe - plain < 64 << 20  # the allocator's granularity; the arrays would be 168 MB
