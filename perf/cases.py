"""The workloads whose speed this repository is judged by, each one pass through the public entry
points of `rbmd_b200`, with a 64-bit answer to compare against.

A case describes a system (`kind` and its size), its options, and what a pass does: `steps` MD steps
of a system that stays on the device followed by the read-back of its state (how an MD program runs
between two outputs), or, with steps = 0, one force evaluation at given positions (the library used
as a force calculator).  Sizes and options are those of the benchmark configurations (LJ fluid 4000,
NaCl 8000, SPC/E 9000, Cu 32,000, the saline serving stream of 1k-64k atoms), of the tests and of
the reference's other options (VERLETLIST, EWALD, NPT).
"""
import math

import numpy as np
import torch

import rbmd_b200
from rbmd_b200 import _abi as A
from rbmd_b200 import synth

PIF = 3.1415927410125732421875  # single-precision pi, the method's constant
PHILOX_GAUSS, PHILOX_ACCEPT = 0x52424531, 0x52424532


# ------------------------------------------------------------------------------------------ cases
def _case(kind, size, steps, precision="fp64", count=1, neighbor="rbl", coulomb="rbe", ensemble="", report=False):
    return dict(kind=kind, size=size, steps=steps, precision=precision, count=count, neighbor=neighbor,
                coulomb=coulomb, ensemble=ensemble, report=report)


def listed():
    return [
        # the smallest run of a unit test or tutorial: 500 LJ atoms, bound by launches
        dict(_case("lj", 5, 20), name="lj_500_fp64"),
        # the LJ fluid configuration: 4000 atoms, plain method, FP64, NVE
        dict(_case("lj", 10, 20), name="lj_4000_fp64"),
        # the molten salt configuration: 8000 ions, RBE with P = 200, Nose-Hoover, FP64
        dict(_case("nacl", 20, 10), name="nacl_8000_fp64"),
        # the rigid water configuration: 3000 SPC/E molecules, SHAKE, mixed precision
        dict(_case("spce", 3000, 10, "mixed"), name="spce_9000_mixed"),
        # the metal configuration: 32,000 Cu atoms, tabulated EAM, mixed precision
        dict(_case("eam", 20, 10, "mixed"), name="eam_32000_mixed"),
        # the serving stream's smallest and largest requests, run alone
        dict(_case("saline", 1200, 10, "mixed"), name="saline_1200_mixed"),
        dict(_case("saline", 64000, 10, "mixed"), name="saline_64000_mixed"),
        # the serving stream: a batch of uneven requests stepped together
        dict(_case("saline", 64000, 10, "mixed", count=64), name="saline_stream_64"),
        # the plain path that the stream is quoted against: one FP64 system per launch
        dict(_case("saline", 4000, 10), name="saline_4000_fp64"),
        # the reference's full method (Verlet neighbours, Ewald sum) with its per-interval energies
        dict(_case("spce", 1500, 5, neighbor="verlet", coulomb="ewald", report=True), name="spce_4500_ewald_fp64"),
        # a force evaluation at positions that come from the host
        dict(_case("saline", 16000, 0, "mixed"), name="forces_saline_16000_mixed"),
        # constant pressure: Berendsen barostat, Verlet neighbours
        dict(_case("lj", 8, 10, neighbor="verlet", ensemble="npt"), name="lj_2048_npt_fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lj", "lj", "nacl", "nacl", "spce", "eam", "saline", "saline", "stream", "alkane", "forces", "ewald",
                       "npt"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "lj":
        return _case("lj", rng.randint(5, 16), rng.randint(8, 24), prec)
    if kind == "nacl":
        return _case("nacl", rng.randint(5, 12) * 2, rng.randint(5, 15), prec)
    if kind == "spce":
        return _case("spce", _log(rng, 330, 12000), rng.randint(4, 10), "mixed")
    if kind == "eam":
        return _case("eam", rng.randint(7, 22), rng.randint(5, 15), prec)
    if kind == "saline":
        return _case("saline", _log(rng, 1000, 64000), rng.randint(4, 10), "mixed")
    if kind == "stream":
        return _case("saline", _log(rng, 2000, 64000), rng.randint(4, 10), "mixed", count=rng.randint(2, 56))
    if kind == "alkane":
        return _case("alkane", rng.randint(3, 9), rng.randint(5, 15), prec)
    if kind == "forces":
        return _case(rng.choice(["saline", "spce"]), _log(rng, 1000, 20000), 0, prec)
    if kind == "ewald":
        return _case("spce", _log(rng, 330, 2500), rng.randint(2, 6), neighbor="verlet", coulomb="ewald", report=True)
    return _case("lj", rng.randint(5, 11), rng.randint(5, 15), neighbor="verlet", ensemble="npt")


def _stream_sizes(case):
    """Log-uniform from 1000 atoms up to `size`, as the serving stream's requests."""
    rng = np.random.default_rng(case["size"] + case["count"])
    return [int(n) for n in np.exp(rng.uniform(math.log(1000), math.log(case["size"]), case["count"]))]


def _systems(case, seed):
    """The systems of a case as synth.SystemData: positions, velocities and parameters from the seed."""
    kw = dict(precision=A.PREC_FP64 if case["precision"] == "fp64" else A.PREC_MIXED)
    if case["neighbor"] == "verlet":
        kw["neighbor"] = A.NEIGH_VERLET
    if case["coulomb"] == "ewald":
        kw["coulomb"] = A.COUL_EWALD
    if case["ensemble"] == "npt":
        kw.update(ensemble=A.ENS_NPT, temp_ctrl=A.TC_BERENDSEN, press_ctrl=A.PC_BERENDSEN, pressure=(0.2, 0.4, 0.5),
                  bulk_modulus=1e4)
    kind, size, seed = case["kind"], case["size"], int(seed) % (1 << 30) + 1
    rng = np.random.default_rng(seed)
    if kind == "lj":
        out = [synth.lj_fcc(cells=size, seed=seed, **kw)]
    elif kind == "nacl":
        out = [synth.nacl_melt(n_side=size, seed=seed, **kw)]
    elif kind == "spce":
        out = [synth.spce_water(n_mol=size, seed=seed, **kw)]
    elif kind == "eam":
        out = [synth.eam_cu(cells=size, seed=seed, build_splines=rbmd_b200.eam_splines, **kw)]
    elif kind == "alkane":
        out = [synth.alkane_chains(n_side=size, seed=seed, **kw)]
    elif case["count"] == 1:
        out = [synth.saline(size, seed=seed, **kw)]
    else:
        out = [synth.saline(n, seed=seed + 7919 * k, **kw) for k, n in enumerate(_stream_sizes(case))]
    if kind in ("lj", "nacl", "eam"):  # thermal displacements: no atom exactly on its lattice site
        for sd in out:
            amp = {"lj": 0.04, "nacl": 0.05, "eam": 0.1}[kind]
            sd.pos = np.mod(sd.pos + rng.normal(scale=amp, size=sd.pos.shape), sd.box_hi)
    return out


def prepare(case, seed):
    sds = _systems(case, seed)
    ctx = rbmd_b200.Context(device=0)
    ids = [ctx.add_system(sd) for sd in sds]
    ctx.init(ids)
    ctx.sync()
    return dict(case=case, ctx=ctx, ids=ids, pos=[sd.pos for sd in sds])


REPORT = ("temperature", "kinetic_energy", "e_lj", "e_coul_near", "e_coul_far", "potential_energy")


def run(state):
    case, ctx, ids = state["case"], state["ctx"], state["ids"]
    if case["steps"] == 0:
        ctx.set_state(ids[0], x=state["pos"][0])
        ctx.compute_forces(ids)
        return ctx.forces(ids[0])
    ctx.step(ids, case["steps"])
    got = [ctx.state(i) for i in ids]
    out = {"x": np.concatenate([g[0] for g in got]), "v": np.concatenate([g[1] for g in got]),
           "image": np.concatenate([g[2] for g in got])}
    if case["report"]:
        t = ctx.thermo(ids[0])
        out["thermo"] = [t[k] for k in REPORT]
    return out


def _atoms(case):
    """Atom count (of the whole batch) for the work estimate."""
    k, s = case["kind"], case["size"]
    n = {"lj": 4 * s ** 3, "nacl": s ** 3, "spce": 3 * s, "eam": 4 * s ** 3, "alkane": 6 * s ** 3, "saline": s}[k]
    if case["count"] > 1:
        n = sum(_stream_sizes(case))
    return n


def work(case):
    """State read and written once per pass; 40 flops per selected pair and, per sampled k, 30 for an
    atom's share of the structure factor and of the force."""
    n = _atoms(case)
    pairs = {"lj": 110, "nacl": 115, "spce": 145, "eam": 45, "alkane": 145, "saline": 145}[case["kind"]]
    ks = {"lj": 0, "nacl": 200, "spce": 100, "eam": 0, "alkane": 100, "saline": 100}[case["kind"]]
    if case["neighbor"] == "verlet":
        pairs, ks = (420, 342) if case["kind"] == "spce" else (55, 0)
    flops = max(1, case["steps"]) * n * (40 * pairs + 60 * ks)
    return {"bytes": n * (2 * (24 + 24 + 12) + 16), "flops": flops}


def tolerance(case):
    """About four times what the pair traversals of this library (which sum in different orders) differ
    by among themselves over two passes of a case's steps."""
    water = case["kind"] in ("spce", "saline")
    if case["steps"] == 0:  # one force evaluation
        return {"rel": 1e-12, "max": 1e-9} if case["precision"] == "fp64" else {"rel": 5e-5, "max": 1e-2}
    if case["precision"] == "fp64":
        # the constraint iteration stops at a change below 1e-5, one round earlier or later by rounding
        return {"rel": 1e-7, "max": 1e-4} if water else {"rel": 1e-11, "max": 1e-8}
    # Mixed precision: 32-bit pair forces part the trajectories by about 1e-7 A within ten steps; a
    # pair nearer to a cut-off than that changes the random-batch picks of its atom, and with them that
    # atom's force.  Seen within 20 steps: 7e-3 of the velocities, 0.4 of the largest.
    return {"rel": 2.8e-2, "max": 0.99, "differ": 1e-4} if water else {"rel": 2e-3, "max": 0.5, "differ": 1e-4}


# ------------------------------------------------------------------------------- the 64-bit answer
def exact(case, seed):
    """The same pass in 64 bits, in plain torch and numpy.  A mixed-precision trajectory is held to its
    positions only: whether a pair at the cut-off counts, and with it the random-batch picks, depends
    on rounding after the first steps; in water, whose light atoms move fastest, that reaches the
    positions too, so there the mixed precision is held to 64 bits by the single force evaluations."""
    water = case["kind"] in ("spce", "saline")
    if case["count"] > 1 or (water and case["precision"] == "mixed" and case["steps"] > 0):
        return None
    n = _atoms(case)
    if n * max(1, case["steps"]) > 700000:
        return None
    m = _Md(_systems(case, seed)[0])
    if case["steps"] == 0:
        m.sort_positions = m.x
        return m.forces().cpu().numpy()
    m.start()
    for _ in range(case["steps"]):
        m.step_once()
    x, v = m.x.cpu().numpy(), (m.v * m.pending[:, None]).cpu().numpy()
    if case["precision"] == "mixed":
        return {"x": x, "v": None, "image": None}
    out = {"x": x, "v": v, "image": m.image.cpu().numpy().astype(np.int32)}
    if case["report"]:
        e = m.energies()
        out["thermo"] = [float(e[k]) for k in REPORT]
    return out


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on arrays of counters (uint64 holding 32-bit words)."""
    m = np.uint64(0xFFFFFFFF)
    c0, c1, c2, c3 = (np.asarray(c, np.uint64) for c in np.broadcast_arrays(c0, c1, c2, c3))
    k0, k1 = np.uint64(k0), np.uint64(k1)
    s32 = np.uint64(32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> s32) ^ c1 ^ k0, p1 & m, (p0 >> s32) ^ c3 ^ k1, p0 & m
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    return c0, c1, c2, c3


def _u01(hi, lo):
    return (((hi >> np.uint64(5)) << np.uint64(26)) | (lo >> np.uint64(6))).astype(np.float64) / 9007199254740992.0


class _Md:
    """One system of the method in 64-bit torch: random-batch or full pair lists over cells, random
    batch or full Ewald, harmonic bonded terms, EAM, water constraints, velocity Verlet with a
    Nose-Hoover chain or Berendsen control."""

    def __init__(self, sd):
        self.sd, self.p = sd, sd.params
        p = self.p
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        T = self.tensor
        self.x, self.n = T(sd.pos), sd.n
        self.v = T(sd.vel) if sd.vel is not None else torch.zeros_like(self.x)
        self.m = T(sd.mass)
        self.q = T(sd.charge) if sd.charge is not None else torch.zeros_like(self.m)
        self.type = T(sd.types).long()
        self.mol = T(sd.molecule).long() if sd.molecule is not None else torch.arange(self.n, device=self.dev)
        self.L = np.asarray(sd.box_hi, np.float64) - np.asarray(sd.box_lo, np.float64)
        self.lo = np.asarray(sd.box_lo, np.float64)
        self.image = torch.zeros_like(self.x)
        self.units = {A.UNITS_LJ: (1.0, 1.0, 1.0, 1.0, 1.0, 1.0),
                      A.UNITS_REAL: (1.9872067e-3, 4.186e-4, 1 / 4.186e-4, 332.06371, 0.0019872067, 68568.415),
                      A.UNITS_METAL: (8.617343e-5, 1.0 / 1.0364269e-4, 1.0364269e-4, 14.399645, 8.617343e-5,
                                      1.6021765e6)}[p.units]
        self.kB, self.fmt2v, self.mvv2e, self.qqr2e, self.boltz, self.nktv2p = self.units
        self.rbl = p.neighbor == A.NEIGH_RBL
        self.rc, self.rs = p.cut_off, p.r_core if self.rbl else p.cut_off
        self.nc = math.ceil(self.rc / self.rs)
        self.eam = p.force_field == A.FF_EAM
        self.coul = p.force_field in (A.FF_LJ_CUT_COUL_LONG, A.FF_CVFF)
        self.special = sd.special_offsets is not None and self.coul
        if self.special:
            off = np.asarray(sd.special_offsets)
            cnt = np.diff(off)
            ids, w = np.full((self.n, cnt.max()), -1), np.ones((self.n, cnt.max()))
            row = np.repeat(np.arange(self.n), cnt)
            col = np.arange(off[-1]) - np.repeat(off[:-1], cnt)
            ids[row, col], w[row, col] = sd.special_ids, sd.special_weights
            self.sp_ids, self.sp_w = T(ids).long(), T(w)
        self.pick_every = 1
        if self.rbl:
            rho = self.n / np.prod(self.L)
            co = 1.0 if self.eam else float(int(np.floor(1.0 + (0.05 / rho - 0.05) + 0.5)))
            num = [int(co * rho * math.ceil(4.0 / 3.0 * PIF * r ** 3) + 1) for r in (self.rs, self.rc)]
            shell = num[1] - num[0]
            self.pick_every = max(1, math.ceil(1.0 / (p.neighbor_sample_num / shell))) if shell > 0 else 1
        self.triples = None
        if p.fix_shake == A.SHAKE_TRUE and sd.angle_atoms is not None:
            self.triples = T(np.asarray(sd.angle_atoms).reshape(-1, 3)).long()
        self.step = 0
        self.pending = torch.ones(self.n, dtype=torch.float64, device=self.dev)

    def tensor(self, a):
        t = torch.as_tensor(np.ascontiguousarray(a), device=self.dev)
        return t.double() if t.is_floating_point() else t

    def box(self):
        return torch.as_tensor(self.L, dtype=torch.float64, device=self.dev)

    def nearest(self, r):
        L = self.box()
        return torch.where(r.abs() > 0.5 * L, r - torch.sign(r) * L, r)

    # ---- pairs
    def pair_blocks(self, x, sort_x, full):
        """Blocks of (i, j, r = image of x_j - x_i, core, picked shell), candidates in the method's order."""
        rc2, rs2 = self.rc ** 2, self.rs ** 2
        nc, dev = self.nc, self.dev
        dims = [max(1, int(self.L[k] / (self.rc / nc))) for k in range(3)]
        d = torch.as_tensor([self.L[k] / dims[k] for k in range(3)], dtype=torch.float64, device=dev)
        dt, lo = torch.as_tensor(dims, device=dev), torch.as_tensor(self.lo, device=dev)
        bin3 = torch.minimum(((sort_x - lo) / d).trunc().long().clamp(min=0), dt - 1)
        cell = bin3[:, 0] + dims[0] * (bin3[:, 1] + dims[1] * bin3[:, 2])
        order = torch.argsort(cell, stable=True)
        counts = torch.bincount(cell, minlength=dims[0] * dims[1] * dims[2])
        starts = torch.cumsum(counts, 0) - counts
        most = int(counts.max())
        slot = torch.arange(self.n, device=dev) - starts[cell[order]]
        table = torch.full((counts.numel(), most), -1, dtype=torch.long, device=dev)
        table[cell[order], slot] = order
        home = ((x - lo) / d).trunc().long()
        a = torch.arange(-nc, nc + 1, device=dev)
        off = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
        size = max(1, int(3e7 // (off.shape[0] * most)))
        for b in range(0, self.n, size):
            i = torch.arange(b, min(self.n, b + size), device=dev)
            at = home[i][:, None, :] + off[None]
            wrapped = torch.remainder(at, dt)
            c = wrapped[..., 0] + dims[0] * (wrapped[..., 1] + dims[1] * wrapped[..., 2])
            j = table[c]
            r = (x[j.clamp(min=0)] - (d * (wrapped - at).double())[:, :, None, :]) - x[i][:, None, None, :]
            j, r = j.reshape(len(i), -1), r.reshape(len(i), -1, 3)
            d2 = r[..., 0] * r[..., 0] + r[..., 1] * r[..., 1] + r[..., 2] * r[..., 2]
            there = j >= 0
            if full:
                core, pick = there & (rc2 - d2 > 1e-4) & (d2 > 1e-4), None
            else:
                shell = there & (rc2 - d2 > 1e-4) & (d2 - rs2 > 1e-4)
                core = there & ~shell & (rs2 - d2 > 1e-4) & (d2 > 1e-4)
                pick = shell & ((torch.cumsum(shell.int(), 1) - 1) % self.pick_every == 0)
            sel = core if pick is None else core | pick
            row, k = sel.nonzero(as_tuple=True)
            yield i[row], j[row, k], self.nearest(r[row, k]), core[row, k]

    def weights(self, i, j):
        if not self.special:
            return 1.0
        w = torch.ones(i.numel(), dtype=torch.float64, device=self.dev)
        for s in range(self.sp_ids.shape[1]):
            w = torch.where(self.sp_ids[i, s] == j, self.sp_w[i, s], w)
        return w

    def lj_terms(self, i, j):
        eps, sig = self.tensor(self.sd.eps), self.tensor(self.sd.sig)
        return torch.sqrt(eps[self.type[i]] * eps[self.type[j]]), ((sig[self.type[i]] + sig[self.type[j]]) / 2) ** 6

    def pair_forces(self, x, sort_x):
        F = torch.zeros_like(x)
        self.virial = torch.zeros(3, dtype=torch.float64, device=self.dev)
        rc2, rs2 = self.rc ** 2, self.rs ** 2
        for i, j, r, core in self.pair_blocks(x, sort_x, not self.rbl):
            d2 = (r * r).sum(1)
            scale = torch.where(core, 1.0, float(self.pick_every))
            e, s6 = self.lj_terms(i, j)
            sd6 = s6 / d2 ** 3
            lj = -24 * e * ((2 * sd6 - 1) * sd6) / d2
            if not self.coul:
                f = lj * scale
                if self.rbl:
                    f = torch.where(self.mol[i] == self.mol[j], 0.0, f)
            else:
                w, a, dis = self.weights(i, j), self.p.alpha, torch.sqrt(d2)
                qq = self.q[i] * self.q[j]
                g = torch.erfc(math.sqrt(a) * dis) / d2 + 2 * math.sqrt(a) * torch.exp(-a * d2) / (math.sqrt(PIF) * dis)
                fc = -qq * g / dis
                if self.rbl:
                    lj = torch.where(core & ~(d2 < rs2), 0.0, lj)
                    f = w * scale * lj + self.qqr2e * scale * fc
                else:
                    f = self.qqr2e * (fc - (1.0 - w) * (-qq / dis ** 3)) + w * lj
            F.index_add_(0, i, f[:, None] * r)
            self.virial += (0.5 * f[:, None] * r * r).sum(0)
        return F

    def eam_row(self, table, r, dr, n):
        rows = self.tensor(np.asarray(table)).reshape(-1, 7)
        p = r / dr + 1.0
        m = p.long().clamp(1, n - 1)
        return rows[m], (p - m).clamp(max=1.0)

    def eam_forces(self, x, sort_x):
        e = self.sd.eam
        rho = torch.zeros(self.n, dtype=torch.float64, device=self.dev)
        blocks = list(self.pair_blocks(x, sort_x, not self.rbl))
        for i, j, r, core in blocks:
            c, p = self.eam_row(e["rhor_spline"], r.norm(dim=1), e["dr"], e["nr"])
            val = ((c[:, 3] * p + c[:, 4]) * p + c[:, 5]) * p + c[:, 6]
            rho.index_add_(0, i, torch.where(core, 1.0, float(self.pick_every)) * val)
        c, p = self.eam_row(e["frho_spline"], rho, e["drho"], e["nrho"])
        fp = (c[:, 0] * p + c[:, 1]) * p + c[:, 2]
        F = torch.zeros_like(x)
        for i, j, r, core in blocks:
            dis = r.norm(dim=1)
            c, p = self.eam_row(e["rhor_spline"], dis, e["dr"], e["nr"])
            z, _ = self.eam_row(e["z2r_spline"], dis, e["dr"], e["nr"])
            rhop = (c[:, 0] * p + c[:, 1]) * p + c[:, 2]
            z2p = (z[:, 0] * p + z[:, 1]) * p + z[:, 2]
            z2 = ((z[:, 3] * p + z[:, 4]) * p + z[:, 5]) * p + z[:, 6]
            psip = fp[i] * rhop + fp[j] * rhop + z2p / dis - z2 / dis ** 2
            f = torch.where(core, 1.0, float(self.pick_every)) * psip / dis
            F.index_add_(0, i, f[:, None] * r)
        return F

    # ---- k space
    def samples(self):
        p, a, P = self.p, self.p.alpha, self.p.coulomb_sample_num
        seed = int(p.seed)
        t = np.arange(4 * P + 256)[:, None]
        dim = np.arange(3)[None]
        g = np.zeros((len(t), 3))
        need = np.ones((len(t), 3), bool)
        for attempt in range(64):
            o = _philox(t, dim | (attempt << 2), self.step, PHILOX_GAUSS, seed & 0xFFFFFFFF, seed >> 32)
            u1, u2 = _u01(o[0], o[1]), _u01(o[2], o[3])
            sigma = np.sqrt(a / 2.0) * self.L / np.pi
            with np.errstate(divide="ignore"):
                val = sigma[None] * np.sqrt(-2.0 * np.log(u1)) * np.cos(2 * np.pi * u2)
            g = np.where(need, val, g)
            need &= u1 < 1e-6
            if not need.any():
                break
        prop = np.copysign(np.floor(np.abs(g) + 0.5), g)
        o = _philox(t, dim, self.step, PHILOX_ACCEPT, seed & 0xFFFFFFFF, seed >> 32)
        u = _u01(o[0], o[1])

        def ratio(m, k):  # target over proposal probability of m in dimension k
            L, sc = self.L[k], math.sqrt(a * self.L[k] ** 2 / np.pi ** 2)
            H = sum(math.exp(-(q * q) * a * L * L) for q in range(-10, 11)) * math.sqrt(a * L * L / np.pi)
            P_m = math.exp(-(2 * np.pi * m / L) ** 2 / (4 * a)) / H
            if m == 0:
                return P_m, math.erf(0.5 / sc)
            return P_m, (math.erf((0.5 + abs(m)) / sc) - math.erf((abs(m) - 0.5) / sc)) / 2

        at, cur, got = 0, None, []
        while len(got) < P:
            new = prop[at]
            if cur is None:
                if np.any(new != 0):
                    cur = new.copy()
                    got.append(cur.copy())
            else:
                for k in range(3):
                    (p1, q1), (p0, q0) = ratio(new[k], k), ratio(cur[k], k)
                    if u[at, k] <= min(1.0, (p1 / p0) * (q0 / q1)):
                        cur[k] = new[k]
                if np.any(cur != 0):
                    got.append(cur.copy())
            at += 1
        return np.array(got)

    def far_forces(self, x):
        a, V, p = self.p.alpha, float(np.prod(self.L)), self.p
        if p.coulomb == A.COUL_RBE:
            m = self.samples()
            H = [sum(math.exp(-(q * q) * a * L * L) for q in range(-10, 11)) * math.sqrt(a * L * L / np.pi) for L in self.L]
            scale = (H[0] * H[1] * H[2] - 1) / p.coulomb_sample_num
        else:
            r = [np.arange(-k, k + 1) for k in p.kmax]
            m = np.stack(np.meshgrid(*r, indexing="ij"), -1).reshape(-1, 3)
            m, scale = m[np.any(m != 0, 1)], 1.0
        k = self.tensor(2 * np.pi * m / self.L)
        k2 = (k * k).sum(1)
        coef = -4 * np.pi / (V * k2)
        if p.coulomb == A.COUL_EWALD:
            coef = coef * torch.exp(-k2 / (4 * a))
        F = torch.zeros_like(x)
        for b in range(0, len(k), 64):
            ph = x @ k[b:b + 64].T
            c, s = torch.cos(ph), torch.sin(ph)
            re, im = self.q @ c, self.q @ s
            F += (coef[b:b + 64] * self.q[:, None] * (c * im - s * re)) @ k[b:b + 64]
        return F * (scale * self.qqr2e)

    # ---- molecules
    def bonded_energy(self, x):
        sd, T = self.sd, self.tensor
        parts = {"bond": x.sum() * 0.0, "angle": x.sum() * 0.0, "dihedral": x.sum() * 0.0}

        def legs(ids, pairs):
            return [self.nearest(x[ids[:, a]] - x[ids[:, b]]) for a, b in pairs]

        if sd.bond_atoms is not None:
            ids, ty = T(np.asarray(sd.bond_atoms).reshape(-1, 2)).long(), T(sd.bond_type).long()
            r, = legs(ids, [(0, 1)])
            parts["bond"] = (T(sd.bond_k)[ty] * (r.norm(dim=1) - T(sd.bond_r0)[ty]) ** 2).sum()
        if sd.angle_atoms is not None:
            ids, ty = T(np.asarray(sd.angle_atoms).reshape(-1, 3)).long(), T(sd.angle_type).long()
            a, b = legs(ids, [(0, 1), (2, 1)])
            th = torch.acos(((a * b).sum(1) / (a.norm(dim=1) * b.norm(dim=1))).clamp(-1, 1))
            parts["angle"] = (T(sd.angle_k)[ty] * (th - T(sd.angle_theta0)[ty] * PIF / 180) ** 2).sum()
        if sd.dihedral_atoms is not None:
            ids, ty = T(np.asarray(sd.dihedral_atoms).reshape(-1, 4)).long(), T(sd.dihedral_type).long()
            b1, b2, b3 = legs(ids, [(0, 1), (2, 1), (3, 2)])
            u, w = torch.linalg.cross(b1, -b2), torch.linalg.cross(b3, -b2)
            phi = torch.atan2(b2.norm(dim=1) * (u * b3).sum(1), (u * w).sum(1))
            sign = torch.where(T(sd.dihedral_sign)[ty] == 1, 1.0, -1.0)
            parts["dihedral"] = (T(sd.dihedral_k)[ty] * (1 + sign * torch.cos(T(sd.dihedral_multiplicity)[ty] * phi))).sum()
        return parts

    def excluded_coulomb(self, x):
        F = torch.zeros_like(x)
        cnt = torch.bincount(self.mol)
        order = torch.argsort(self.mol, stable=True)
        first = torch.cumsum(cnt, 0) - cnt
        for k in range(int(cnt.max())):
            big = (cnt[self.mol] >= 3) & (k < cnt[self.mol])
            i = big.nonzero()[:, 0]
            j = order[first[self.mol[i]] + k]
            i, j = i[i != j], j[i != j]
            r = self.nearest(x[i] - x[j])
            fc = -332.06371 * self.q[i] * self.q[j] / r.norm(dim=1) ** 3
            F.index_add_(0, i, ((1.0 - self.weights(i, j)) * fc)[:, None] * r)
        return F

    def forces(self):
        x = self.x
        F = self.eam_forces(x, self.sort_positions) if self.eam else self.pair_forces(x, self.sort_positions)
        if self.rbl:
            F = F - F.mean(0)
        if self.coul:
            F = F + self.far_forces(x)
        if self.p.force_field == A.FF_CVFF:
            if self.rbl and self.special:
                F = F + self.excluded_coulomb(x)
            y = x.clone().requires_grad_(True)
            F = F - torch.autograd.grad(sum(self.bonded_energy(y).values()), y)[0]
        return F

    # ---- integration
    def temperature_of(self, v):
        s = float((self.m[:, None] * v * v).sum()) * self.mvv2e
        dof = 3 * self.n - 3 - (self.n if self.p.fix_shake == A.SHAKE_TRUE else 0)
        if self.p.fix_shake == A.SHAKE_FALSE:
            dof = 3 * self.n
        self.tsum = s
        return 0.5 * s / (dof * self.kB / 2.0)

    def start(self):
        self.sort_positions = self.x
        self.F = self.forces()
        self.T = self.temperature_of(self.v)
        self.dof = 3.0 * self.n - 3 - (self.n if self.p.fix_shake == A.SHAKE_TRUE else 0)
        self.eta_dot, self.eta_dd = [0.0] * 4, [0.0] * 3
        self.eta_dd[1] = self.eta_dd[2] = -1 / self.p.temperature[2] ** 2

    def chain_half(self):
        dt, boltz, t, f = self.p.timestep, self.boltz, self.p.temperature[0], 1 / self.p.temperature[2]
        mass = [self.dof * boltz * t / (f * f)] + [boltz * t / (f * f)] * 2
        e, dd = self.eta_dot, self.eta_dd
        target = self.dof * boltz * t
        dd[0] = (self.dof * boltz * self.T - target) / mass[0]
        for c in (2, 1, 0):
            g = math.exp(-0.125 * dt * e[c + 1])
            e[c] = (e[c] * g + dd[c] * 0.25 * dt) * g
        factor = math.exp(-0.5 * dt * e[0])
        self.T *= factor * factor
        dd[0] = (self.dof * boltz * self.T - target) / mass[0]
        e[0] = (e[0] * g + dd[0] * 0.25 * dt) * g
        for c in (1, 2):
            g = math.exp(-0.125 * dt * e[c + 1])
            e[c] *= g
            dd[c] = (mass[c - 1] * e[c - 1] * e[c - 1] - boltz * t) / mass[c]
            e[c] = (e[c] + dd[c] * 0.25 * dt) * g
        return factor

    def wrap(self, x, closed=False):
        lo, L = torch.as_tensor(self.lo, device=self.dev), self.box()
        low = x < lo
        high = (x > lo + L) if closed else (x >= lo + L)
        self.image = self.image - low.double() + (high & ~low).double()
        return torch.where(low, x + L, torch.where(high, x - L, x))

    def step_once(self):
        p, dt, c = self.p, self.p.timestep, self.fmt2v
        self.step += 1
        scale = self.chain_half() if p.temp_ctrl == A.TC_NOSE_HOOVER else 1.0
        v0 = self.v * self.pending[:, None] * scale
        self.pending = torch.ones_like(self.pending)
        acc = self.F / self.m[:, None] * c
        x0 = self.x
        v = v0 + 0.5 * dt * acc
        x = self.wrap(x0 + v * dt)
        self.sort_positions = x
        if self.triples is not None:
            x, v = self.shake(x0, v0, acc, x, v)
        self.x = x
        self.F = self.forces()
        acc = self.F / self.m[:, None] * c
        v1 = v + 0.5 * dt * acc
        self.T = self.temperature_of(v1)
        if p.temp_ctrl == A.TC_NOSE_HOOVER:
            f = self.chain_half()
            if self.triples is None:
                self.pending = self.pending * f
            else:
                self.pending = torch.where(torch.isin(torch.arange(self.n, device=self.dev), self.triples.reshape(-1)),
                                           1.0, f * self.pending)
        elif p.temp_ctrl == A.TC_BERENDSEN:
            self.pending = self.pending * math.sqrt(1.0 + dt / p.temperature[2] * (p.temperature[0] / self.T - 1.0))
        if self.triples is not None:
            v1 = self.rattle(v1)
        self.v = v1
        if p.ensemble == A.ENS_NPT:
            vir = float(self.virial.sum())
            press = (self.dof * self.boltz * self.T + vir) / 3.0 / float(np.prod(self.L)) * self.nktv2p
            goal = p.pressure[0] + self.step / p.num_steps * (p.pressure[1] - p.pressure[0])
            mu = (1.0 - dt / p.pressure[2] * (goal - press) / p.bulk_modulus) ** (1.0 / 3.0)
            lo, L = torch.as_tensor(self.lo, device=self.dev), self.box()
            inner = (self.x - lo) / L
            mid = self.lo + 0.5 * self.L
            self.lo, self.L = mid - 0.5 * mu * self.L, mu * self.L
            self.x = self.wrap(inner * self.box() + torch.as_tensor(self.lo, device=self.dev))

    def triple_legs(self, x):
        t = self.triples
        return [self.nearest(x[t[:, a]] - x[t[:, b]]) for a, b in ((1, 0), (2, 1), (0, 2))]

    def shake(self, x0, v0, acc, x, v):
        """Bond lengths 1, 1 and the chord of 109.47 degrees held by the method's iteration: linear
        solves with the quadratic terms of the previous iterate, until no multiplier moves by 1e-5."""
        t, dt = self.triples, self.p.timestep
        free = x0 + v0 * dt + 0.5 * dt * dt * acc
        im = 1.0 / self.m[t]
        r = self.triple_legs(x0)
        s = [self.nearest(free[t[:, a]] - free[t[:, b]]) for a, b in ((0, 1), (1, 2), (2, 0))]
        # how multiplier b moves leg a: the leg's atoms gain +-r_b / m
        zero = torch.zeros_like(im[:, 0])
        gain = [[im[:, 0] + im[:, 1], -im[:, 1], -im[:, 0]],
                [-im[:, 1], im[:, 1] + im[:, 2], -im[:, 2]],
                [-im[:, 0], -im[:, 2], im[:, 0] + im[:, 2]]]
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        mat = torch.stack([torch.stack([2 * gain[a][b] * dot(s[a], r[b]) for b in range(3)], -1) for a in range(3)], 1)
        chord = math.sqrt(2.0 - 2.0 * math.cos(109.47 / 180.0 * PIF))
        want = [1.0, 1.0, chord * chord]
        lam = torch.zeros(len(t), 3, dtype=torch.float64, device=self.dev)
        live = torch.ones(len(t), dtype=torch.bool, device=self.dev)
        inv = torch.linalg.inv(mat)
        for _ in range(5000):
            rhs = []
            for a in range(3):
                move = sum((gain[a][b] * lam[:, b])[:, None] * r[b] for b in range(3))
                rhs.append(want[a] - dot(s[a], s[a]) - dot(move, move) + zero)
            new = (inv @ torch.stack(rhs, -1)[..., None])[..., 0]
            still = (new - lam).abs().max(1).values > 1e-5
            lam = torch.where(live[:, None], new, lam)
            live = live & still
            if not bool(live.any()):
                break
        push = torch.stack([lam[:, :1] * r[0] * im[:, :1] - lam[:, 2:] * r[2] * im[:, :1],
                            lam[:, 1:2] * r[1] * im[:, 1:2] - lam[:, :1] * r[0] * im[:, 1:2],
                            lam[:, 2:] * r[2] * im[:, 2:] - lam[:, 1:2] * r[1] * im[:, 2:]], 1)
        flat = t.reshape(-1)
        whole, vnew = x0.clone(), v.clone()
        whole[flat] = (free[t] + push).reshape(-1, 3)
        vnew[flat] = (v[t] + push / dt).reshape(-1, 3)
        held = torch.zeros(self.n, dtype=torch.bool, device=self.dev)
        held[flat] = True
        drifted = self.image  # the method counts the constrained crossing on top of the drift's
        xs = self.wrap(whole, closed=True)
        self.image = torch.where(held[:, None], self.image, drifted)
        return torch.where(held[:, None], xs, x), vnew

    def rattle(self, v):
        t = self.triples
        im = 1.0 / self.m[t]
        r = self.triple_legs(self.x)
        dv = [v[t[:, a]] - v[t[:, b]] for a, b in ((0, 1), (1, 2), (2, 0))]
        dot = lambda a, b: (a * b).sum(1)  # noqa: E731
        gain = [[im[:, 0] + im[:, 1], -im[:, 1], -im[:, 0]],
                [-im[:, 1], im[:, 1] + im[:, 2], -im[:, 2]],
                [-im[:, 0], -im[:, 2], im[:, 0] + im[:, 2]]]
        mat = torch.stack([torch.stack([gain[a][b] * dot(r[a], r[b]) for b in range(3)], -1) for a in range(3)], 1)
        rhs = torch.stack([-dot(dv[a], r[a]) for a in range(3)], -1)
        lam = torch.linalg.solve(mat, rhs[..., None])[..., 0]
        push = torch.stack([lam[:, :1] * r[0] * im[:, :1] - lam[:, 2:] * r[2] * im[:, :1],
                            lam[:, 1:2] * r[1] * im[:, 1:2] - lam[:, :1] * r[0] * im[:, 1:2],
                            lam[:, 2:] * r[2] * im[:, 2:] - lam[:, 1:2] * r[1] * im[:, 2:]], 1)
        out = v.clone()
        out[t.reshape(-1)] = (v[t] + push).reshape(-1, 3)
        return out

    def energies(self):
        """Per-atom energies of the current positions, as the thermo output reports them."""
        n, a, p = self.n, self.p.alpha, self.p
        lj = near = 0.0
        for i, j, r, _ in self.pair_blocks(self.x, self.x, True):
            d2 = (r * r).sum(1)
            e, s6 = self.lj_terms(i, j)
            w, dis = self.weights(i, j), torch.sqrt(d2)
            sd6 = s6 / d2 ** 3
            lj += float((w * 0.5 * 4 * e * (sd6 - 1) * sd6).sum())
            qq = 0.5 * self.q[i] * self.q[j] / dis
            near += self.qqr2e * float((qq * torch.erfc(math.sqrt(a) * dis) - (1.0 - w) * qq).sum())
        r = [np.arange(-k, k + 1) for k in p.kmax]
        m = np.stack(np.meshgrid(*r, indexing="ij"), -1).reshape(-1, 3)
        k = self.tensor(2 * np.pi * m[np.any(m != 0, 1)] / self.L)
        k2 = (k * k).sum(1)
        ph = self.x @ k.T
        rho2 = (self.q @ torch.cos(ph)) ** 2 + (self.q @ torch.sin(ph)) ** 2
        far = float((torch.exp(-k2 / (4 * a)) / k2 * rho2).sum()) * 2 * np.pi / float(np.prod(self.L)) * self.qqr2e / n
        far -= math.sqrt(a / np.pi) * float((self.q * self.q).sum()) / n * self.qqr2e
        b = {q: float(t) for q, t in self.bonded_energy(self.x).items()}
        sd = self.sd
        extra = b["bond"] / len(sd.bond_type) + b["angle"] / len(sd.angle_type)
        return dict(temperature=self.T, kinetic_energy=self.tsum / n * 0.5, e_lj=lj / n, e_coul_near=near / n,
                    e_coul_far=far, potential_energy=lj / n + far + near / n + extra)
