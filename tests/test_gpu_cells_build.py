"""Cell lists where the build kernel's branches part: cells with more atoms than a bucket holds (their
chains), boxes of more cells than are added up in one level, boxes of a few cells, and lists
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


def _cells_ms(ctx_factory, sd):
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    ctx.init(sid)
    ctx.step(sid, 2)
    ctx.profile(True)
    ctx.step(sid, 5)
    ctx.sync()
    return ctx.profile_get("cells")[0]


def test_cost_does_not_grow_with_other_cells_overflow(ctx_factory):
    """A liquid slab in a box of ten times its volume: most cells that hold atoms hold more than a bucket.
    An atom is compared with its own cell's atoms only, so the list costs about what it costs in the full
    box, not atoms times overflow (4 ms per list for these 9000 atoms)."""
    full = synth.saline(9000, seed=3)
    slab = full.copy()
    slab.box_hi = full.box_hi * [1, 1, 10]
    assert _cells_ms(ctx_factory, slab) < 10 * _cells_ms(ctx_factory, full)


@pytest.mark.parametrize("batch", [False, True], ids=["alone", "with_large_and_small_box"])
def test_lists_built_by_every_route_in_turn(ctx_factory, oracle_mod, batch):
    """Over-full cells, lists built by the drift kernel's binning (steps), the standalone count (cells) and
    the static list call one after the other: the two count buffers and the chains stay in step."""
    rng = np.random.default_rng(5)
    sd = synth.lj_fcc(cells=6, precision=A.PREC_FP64, r_core=2.5)  # cells of 13 atoms, buckets of 8
    sd.box_hi = sd.box_hi * [1, 1, 8]

    def sparse(n, box, side):
        g = np.stack(np.meshgrid(*[np.arange(side)] * 3), -1).reshape(-1, 3)
        other = synth.SystemData((rng.permutation(g)[:n] + 0.5) * box / side, np.ones(n), np.zeros(n), sd.eps, sd.sig,
                                 [0, 0, 0], [box] * 3, params=A.Params.from_buffer_copy(sd.params))
        return other

    ctx = ctx_factory()
    ids = [ctx.add_system(sd)]
    if batch:
        ids.append(ctx.add_system(sparse(500, 80.0, 16)))  # 32,768 cells
        ids.append(ctx.add_system(sparse(40, 7.6, 4)))     # 27
    ctx.init(ids)

    def check():
        x, _, _ = ctx.state(ids[0])
        now = sd.copy()
        now.pos = x
        o = oracle_mod.Oracle(now)
        for a, b in zip(ctx.cells(ids[0]), o.cells()):
            assert np.array_equal(a, b)
        nc, ns, lists = ctx.rbl_lists_static(ids[0], 512)
        o_nc, o_ns, o_ids = o.rbl_lists(512)
        assert np.array_equal(nc, o_nc) and np.array_equal(ns, o_ns)
        for i in range(sd.n):
            k = nc[i] + ns[i]
            assert np.array_equal(np.sort(lists[i, :k]), np.sort(o_ids[i, :k]))

    check()
    for _ in range(3):
        ctx.step(ids, 1)
        check()
        ctx.step(ids, 2)
        ctx.thermo(ids[0])
        check()


@pytest.mark.parametrize("edge", [80, 81])  # 512,000 cells: groups; 531,441: groups of groups
def test_cells_of_a_huge_box_match_oracle(ctx_factory, oracle_mod, edge):
    rng = np.random.default_rng(edge)
    box = 2.5 * edge + 0.01
    sd = _lj(5000, box, rng.uniform(0, box, (5000, 3)))
    sd.params.r_core = 2.5
    ctx = ctx_factory()
    sid = ctx.add_system(sd)
    for _ in range(3):
        for a, b in zip(ctx.cells(sid), oracle_mod.Oracle(sd).cells()):
            assert np.array_equal(a, b)
        sd.pos = rng.uniform(0, box, (5000, 3))
        ctx.set_state(sid, x=sd.pos)


def test_cost_of_a_huge_box_is_linear(ctx_factory):
    """64 times the cells for 200,000 atoms: at most 160 times the time (the sums before a block's cells
    went up with the square of the cells: 1400 times)."""
    def gas(edge):
        g = np.stack(np.meshgrid(*[np.arange(59)] * 3), -1).reshape(-1, 3)[:200000]
        sd = _lj(200000, 2.5 * edge + 0.1, (g + 0.5) * (2.5 * edge / 59))
        sd.params.r_core = 2.5
        return sd
    assert _cells_ms(ctx_factory, gas(400)) < 160 * _cells_ms(ctx_factory, gas(100))
