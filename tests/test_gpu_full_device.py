"""States and forces of a system on a device whose memory is used up: reading and writing them must not
need device memory."""
import numpy as np
import pytest
import torch

from rbmd_b200 import _abi as A
from rbmd_b200 import synth

pytestmark = pytest.mark.gpu


def test_state_crosses_without_device_memory(ctx_factory):
    n_side = 200
    n = n_side ** 3  # 192 MB per array of three components
    g = np.arange(n_side) * 1.2 + 0.6
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(0)
    vel = rng.normal(size=(n, 3))
    p = A.default_params(force_field=A.FF_LJ_CUT, neighbor=A.NEIGH_RBL, cut_off=2.4, r_core=2.4,
                         neighbor_sample_num=100, units=A.UNITS_LJ, timestep=0.001, temp_ctrl=A.TC_NONE)
    sd = synth.SystemData(pos, np.ones(n), np.zeros(n), [1.0], [1.0], [0, 0, 0], [1.2 * n_side] * 3, vel=vel, params=p)
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.compute_forces(sid)
    small = ctx.add_system(synth.lj_fcc(cells=4))  # every kernel involved is loaded
    ctx.set_state(small, *ctx.state(small))
    hold = []
    for size in (1 << 30, 1 << 26):  # all but the last 64 MB
        while torch.cuda.mem_get_info()[0] > size + (64 << 20):
            free = torch.cuda.mem_get_info()[0]
            try:
                hold.append(torch.empty(max(size, (free - (64 << 20)) // 2), dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                break
    try:
        x, v, img = ctx.state(sid)
        assert np.array_equal(x, pos) and np.array_equal(v, vel) and not img.any()
        forces = ctx.forces(sid)
        ctx.set_state(sid, x=pos[::-1], v=-vel)
        x, v, _ = ctx.state(sid)
        assert np.array_equal(x, pos[::-1]) and np.array_equal(v, -vel)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.isfinite(forces).all() and np.array_equal(forces, ctx.forces(sid))
