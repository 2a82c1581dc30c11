"""What a user of the engine has it do, as timed cases.

Every case goes through the public entry points (moleculardynamics_gb300/engine.py over
include/mdgb.h).  A run uploads its start state, begins, steps and hands back what that run is
made for: the FP64 forms the whole FP64 state (and the energy records, where the run writes
them), the precision form the animation frame of its last step, in the FP32 layout of the
reference's .anm file.  Sizes are those of the benchmark's systems and of the tests.
"""
import math

import numpy as np
import torch

from moleculardynamics_gb300 import engine as eng
from moleculardynamics_gb300 import lattice as lat

RS, RC = 9.534, 8.5125            # LJ list radius and cutoff: 2.8 and 2.5 sigma of argon
MB_RS, MB_RC = 3.5, 3.0           # bond-order list radius and cutoff
DIAMOND_A = 4 * 1.5 / math.sqrt(3.0)


def listed():
    return [
        # The smallest system of the benchmark set, 864 argon atoms in a periodic box, plain FP64:
        # where each launch and each dependent chain shows.
        dict(name="lj64_864", kind="lj64", cells=6, periodic=True, steps=100, dt=2.0, records=50),
        # 8,000 argon atoms in the reference's own walls, plain FP64, as cpumd runs them.
        dict(name="lj64_walls_8000", kind="lj64", cells=13, atoms=8000, periodic=False, steps=100,
             dt=2.0, records=50),
        # Plain FP64 at scale: what the precision form is compared with (108,000 atoms).
        dict(name="lj64_108k", kind="lj64", cells=30, periodic=True, steps=10, dt=2.0, records=0),
        # The reference's own use: N and O bond-order atoms beside neon, both potentials, walls.
        dict(name="both64_172", kind="both64", cells=2, neon=3, steps=100, dt=0.5, records=50),
        # The benchmark set's bond-order system, 4,096 N atoms on a diamond lattice, plain FP64.
        dict(name="bo64_4096", kind="bo64", cells=8, periodic=False, oxygen=False, steps=20,
             dt=0.5),
        # A small system in the precision form, untuned, for long runs: latency counts.
        dict(name="lj32_4000", kind="lj32", cells=10, steps=200, dt=2.0, tune=False),
        # The headline system: 1,048,576 argon atoms, precision form, tiles tuned beforehand.
        dict(name="lj32_1m", kind="lj32", cells=64, steps=100, dt=2.0, tune=True),
        # The batched form: 256 replicas of 256 to 32,000 atoms in one context, tuned.
        dict(name="batch_256", kind="batch", replicas=256, nmin=256, nmax=32000, sizes=4096,
             steps=60, dt=2.0, tune=True),
        # The precision form of the bond order on 32,768 N atoms.
        dict(name="bo32_32k", kind="bo32", cells=16, oxygen=False, temperature=900.0, steps=50,
             dt=0.5),
        # The same lattice driven by the learned direct-force head, checked every 10 steps.
        dict(name="surrogate_32k", kind="surrogate", cells=16, temperature=900.0, steps=20, dt=0.5,
             hidden=64),
        # Force matching of the energy network on one configuration of that size (tensor cores,
        # forward and backward): Adam steps.
        dict(name="train_32k", kind="train", cells=16, temperature=900.0, steps=10),
        # The reference's functions called one by one on host arrays, as a program that keeps
        # cpumd's own loop calls them: one step of 864 atoms with its list build.
        dict(name="calls_864", kind="calls", cells=6),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges (partly filled lattices give odd atom counts)."""
    kind = rng.choice(["lj64", "lj64", "both64", "bo64", "lj32", "lj32", "batch", "bo32",
                       "surrogate", "train", "calls"])
    if kind == "lj64":
        periodic = rng.random() < 0.5
        cells = int(round(_log(rng, 6, 30)))
        lo = 4 * (cells - 1) ** 3 if cells > 6 else 640
        steps = 100 if cells < 14 else 10
        return dict(kind=kind, cells=cells, atoms=rng.randint(lo, 4 * cells ** 3),
                    periodic=periodic, steps=steps, dt=2.0,
                    records=rng.choice([0, 50]) if steps == 100 else 0)
    if kind == "both64":
        return dict(kind=kind, cells=rng.randint(2, 5), neon=rng.randint(3, 8),
                    steps=rng.randint(40, 100), dt=0.5, records=50)
    if kind == "bo64":
        periodic = rng.random() < 0.5
        return dict(kind=kind, cells=rng.randint(5 if periodic else 3, 8), periodic=periodic,
                    oxygen=rng.random() < 0.5, steps=rng.randint(10, 20), dt=0.5)
    if kind == "lj32":
        cells = int(round(_log(rng, 8, 64)))
        return dict(kind=kind, cells=cells, atoms=4 * rng.randint((cells - 1) ** 3, cells ** 3),
                    steps=rng.randint(100, 200) if cells < 24 else rng.randint(50, 100), dt=2.0,
                    tune=rng.random() < 0.5)
    if kind == "batch":
        nmax = int(_log(rng, 2000, 32000))
        return dict(kind=kind, replicas=int(_log(rng, 16, 256)), nmin=256, nmax=nmax,
                    sizes=rng.randint(1, 10 ** 6), steps=rng.randint(40, 60), dt=2.0,
                    tune=rng.random() < 0.5)
    if kind == "bo32":
        return dict(kind=kind, cells=int(round(_log(rng, 5, 16))), oxygen=rng.random() < 0.5,
                    temperature=rng.choice([300.0, 900.0]), steps=rng.randint(20, 50), dt=0.5)
    if kind == "surrogate":
        return dict(kind=kind, cells=int(round(_log(rng, 6, 16))), temperature=900.0,
                    steps=rng.randint(15, 20), dt=0.5, hidden=rng.choice([32, 64, 128]))
    if kind == "train":
        return dict(kind=kind, cells=int(round(_log(rng, 6, 16))),
                    temperature=rng.choice([300.0, 900.0]), steps=rng.randint(8, 10))
    cells = rng.randint(5, 9)
    return dict(kind=kind, cells=cells, atoms=rng.randint(4 * (cells - 1) ** 3, 4 * cells ** 3))


# ------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """(pos4, vel3, box edge, bond-order atoms, mass table) of a case, on the host."""
    kind = case["kind"]
    if kind in ("lj64", "lj32", "calls"):
        noise = 0.05 if kind == "calls" else 0.0
        pos, vel, L = lat.make_system("fcc", case["cells"], 94.4, seed=seed, noise=noise,
                                      natoms=case.get("atoms"))
        return pos, vel, L, 0, "argon"
    if kind == "both64":
        p1, v1, _ = _diamond(case["cells"], 300.0, seed, True)
        p2, v2, _ = lat.make_system("fcc", case["neon"], 100.0, seed=seed + 1, a=6.0,
                                    species=lat.SPECIES_NG, mass_table="neon")
        # side by side, three angstrom apart
        p2[:, 0] += p1[:, 0].max() - p2[:, 0].min() + 3.0
        return (np.concatenate([p1, p2]), np.concatenate([v1, v2]), 0.0, len(p1), "neon")
    pos, vel, L = _diamond(case["cells"], case.get("temperature", 300.0), seed,
                           case.get("oxygen", False))
    return pos, vel, L, len(pos), "neon"


def _diamond(cells, temperature, seed, oxygen):
    pos, vel, L = lat.make_system("diamond", cells, temperature, seed=seed, a=DIAMOND_A,
                                  noise=0.02, species=lat.SPECIES_N, mass_table="neon")
    if oxygen:
        pos[::2, 3] = lat.SPECIES_O
    return pos, vel, L


def _pinned(a):
    p = eng.pinned(a.shape, a.dtype)
    p[...] = a
    return p


def _ensemble(case, seed):
    """(pos4, vel3, atoms and box edge per replica); whole groups of four atoms in all, which is
    how the animation frames are laid out.  The sizes are the case's own, the velocities the
    seed's."""
    pos, vel, natoms, boxes, temps = lat.make_batch(case["replicas"], case["nmin"], case["nmax"],
                                                    seed=case["sizes"])
    spare = int(natoms.sum()) % 4
    natoms[-1] -= spare
    rng, a = np.random.default_rng(seed), 0
    for n, t in zip(natoms, temps):
        vel[a:a + n] = lat.maxwell_boltzmann(rng, np.full(n, lat.MASS["argon"][2]), float(t))
        a += n
    return pos[:a].copy(), vel[:a].copy(), natoms, boxes


def _config(case, n, L, nmb, table):
    kind = case["kind"]
    periodic = case.get("periodic", kind in ("lj32", "bo32", "surrogate", "train"))
    return eng.make_config(
        n_lj=n - nmb, n_mb=nmb, dt=case.get("dt", 0.5), lj_rs=RS, lj_rcut=RC, mb_rs=MB_RS,
        mb_rcut=MB_RC, use_lj=int(nmb < n), use_mb=int(nmb > 0),
        output_timesteps=case.get("records", 0), periodic=int(periodic),
        box=L if periodic else 0.0,
        precision=eng.PREC_MIXED if kind in ("lj32", "bo32", "surrogate") else eng.PREC_FP64,
        species=eng.SPECIES_ARGON if table == "argon" else eng.SPECIES_NEON)


def _head(hidden, seed):
    """Seeded weights of a direct-force head, W1 [h][32], b1, W2 [h][h], b2, W3 [32][h], b3."""
    rng = np.random.default_rng(seed)
    part = [rng.standard_normal((hidden, 32)) / math.sqrt(32), 0.1 * rng.standard_normal(hidden),
            rng.standard_normal((hidden, hidden)) / math.sqrt(hidden),
            0.1 * rng.standard_normal(hidden),
            rng.standard_normal((32, hidden)) / math.sqrt(hidden), 0.1 * rng.standard_normal(32)]
    return np.concatenate([p.ravel() for p in part]).astype(np.float32)


# normalisation of the descriptors of the diamond lattice at 300 to 900 K
DESC_MEAN, DESC_ISTD, HEAD_SCALE = 1.5, 1.0, 1.0e-3


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "batch":
        pos, vel, natoms, boxes = _ensemble(case, seed)
        cfg = eng.make_config(dt=case["dt"], lj_rs=RS, lj_rcut=RC, precision=eng.PREC_MIXED,
                              periodic=1, species=eng.SPECIES_ARGON)
        s["engine"] = e = eng.Batch(cfg, natoms, boxes)
    else:
        pos, vel, L, nmb, table = _inputs(case, seed)
        if kind == "calls":
            box = 2.0 * float(np.abs(pos[:, :3]).max())
            s.update(shim=eng.Shim(eng.SPECIES_ARGON), pos=pos, vel=vel, box=box)
            return s
        s["engine"] = e = eng.Engine(_config(case, len(pos), L, nmb, table))
    if kind == "train":
        e.upload(pos, vel)
        e.begin(0.0)
        s["model"] = m = eng.Surrogate(seed=seed, cutoff=3.0)
        m.collect(e)
        return s
    # a long run keeps its transfer buffers page-locked
    s["pos"], s["vel"] = _pinned(pos), _pinned(vel)
    if kind == "surrogate":
        s["model"] = m = eng.Surrogate(seed=seed, cutoff=3.0)
        m.set_model(1, case["hidden"])
        m.normalisation(np.full(32, DESC_MEAN), np.full(32, DESC_ISTD))
        m.head_params(_head(case["hidden"], seed))
        m.head_scale(HEAD_SCALE)
        m.attach(e, 1e30, 10)
    if kind in ("lj32", "batch", "bo32", "surrogate"):
        # the frame of the run's last step
        e.set_animation(case["steps"] - 1, 2)
        s["out"] = (np.zeros((e.n, 4), np.float32), np.zeros((e.n, 3), np.float32))
    else:
        s["out"] = (eng.pinned((e.n, 4)), eng.pinned((e.n, 3)))
    if case.get("tune"):
        # tiles picked on a state that has left the lattice, as a program does once per system
        e.upload(s["pos"], s["vel"])
        e.begin(0.0)
        e.step(60)
        e.autotune(3)
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "calls":
        return _calls(state)
    e = state["engine"]
    if kind == "train":
        m = state["model"]
        m.train_forces(case["steps"], lr=1e-3, w_energy=0.1, w_force=1.0)
        return m.params()
    lib, h = e.lib, e.h
    e._ck(lib.md_upload(h, state["pos"], state["vel"]), "md_upload")
    e.begin(0.0)
    e.step(case["steps"])
    pos, vel = state["out"]
    if kind in ("lj32", "batch", "bo32", "surrogate"):
        e._ck(lib.md_get_animation_frame(h, e.animation_count() - 1, pos.ctypes.data,
                                         vel.ctypes.data), "md_get_animation_frame")
        return {"pos": pos, "vel": vel}
    e._ck(lib.md_download(h, pos, vel), "md_download")
    out = {"pos": pos, "vel": vel}
    if case.get("records"):
        out["records"] = e.records()
    return out


def _calls(state):
    """One iteration of cpumd's loop through the reference-signature functions."""
    sh, pos, vel = state["shim"], state["pos"].copy(), state["vel"].copy()
    n = len(pos)
    a, b, c = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros((n, 3))
    rows, nls, nlargest = sh.build_neighbor_list(pos, RS, RC, state["box"])
    rcutsq = float(np.float32(float(np.float32(RC)) ** 2))
    f = sh.lennard_jones_forces(pos, rows, nlargest, rcutsq)
    a[:] = sh.calculate_accelerations(pos, f)
    sh.predict(pos, vel, a, b, c, 2.0)
    f = sh.lennard_jones_forces(pos, rows, nlargest, rcutsq)
    sh.correct(pos, vel, f, a, b, c, 2.0, n ** (1.0 / 3.0) * 52.8)
    thermo = sh.perform_calculations(pos, vel)
    return {"rows": rows, "force": f, "pos": pos, "vel": vel, "acc": a, "b": b, "c": c,
            "thermo": thermo}


# -------------------------------------------------------------------- work
def _natoms(case):
    kind = case["kind"]
    if kind == "batch":
        # mean of a log-uniform draw
        return case["replicas"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] /
                                                                           case["nmin"])
    if kind in ("lj64", "lj32", "calls"):
        return case.get("atoms", 4 * case["cells"] ** 3)
    return 8 * case["cells"] ** 3


def work(case):
    """Bytes and operations that a pass cannot do without.  LJ: 75 list entries within 2.8 sigma
    and 54 pairs within 2.5 sigma per atom; 8 operations for the distance of an entry, 20 for a
    pair's force, 53 for the Gear update; the state (position 32, four derivatives of 24 bytes)
    read and written once a step, a 2-byte list entry read once.  Bond order: 28 neighbours,
    75 operations a pair, 60 for a triplet's angle terms; descriptors 20 per function and
    neighbour pair."""
    kind, n = case["kind"], _natoms(case)
    if kind == "calls":
        return {"bytes": n * (4 * 128 + 4 * 700 + 300), "flops": n * 2 * (75 * 8 + 54 * 20)}
    steps = case["steps"]
    if kind == "train":
        net = 2 * (32 * 64 + 64 * 64 + 64)
        return {"bytes": n * steps * (28 * 16 + 32 + 32 * 8),
                "flops": n * steps * (12 * net + 2 * 378 * 16 * 20)}
    flops = n * steps * 53.0
    nbytes = n * steps * 2.0 * 128
    if kind in ("lj64", "lj32", "batch"):
        flops += n * steps * (75 * 8 + 54 * 20)
        nbytes += n * steps * 75 * 2
    elif kind == "surrogate":
        flops += n * steps * (378 * 16 * 20 + 28 * 16 * 8 + 2 * (64 * 32 + case["hidden"] ** 2))
        nbytes += n * steps * 28 * 4
    else:
        flops += n * steps * (28 * 75 + 28 * 27 * 60)
        nbytes += n * steps * 28 * 4
    if kind == "both64":
        m = 4 * case["neon"] ** 3
        flops += m * steps * (20 * 28 + 53)
        nbytes += m * steps * (256 + 40)
    return {"bytes": nbytes + 2 * 56 * n, "flops": flops}


# ------------------------------------------- the same runs in 64-bit torch
F32 = np.float32


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _tens(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


class _Cells:
    """Build-time cells of one list: which pairs are candidates of one another."""

    def __init__(self, x, rs, L):
        rs = float(F32(rs))
        if L:
            cells = int(math.floor(L / rs))
            self.cells, half, cs = (cells if cells >= 3 else 1), L * 0.5, 0.0
            cs = L / self.cells
        else:
            box = float(x.abs().max()) * 2
            self.cells, half, cs = max(1, int(box / rs + float(F32(0.99)))), box / 2, rs
        c = torch.floor((x + half) / cs).to(torch.int64)
        self.c = c.clamp(0, self.cells - 1) if L else c
        self.L = L

    def adjacent(self, i, j):
        """j is a candidate in i's row."""
        if self.L and self.cells == 1:
            return torch.ones_like(i, dtype=torch.bool)
        d = self.c[j] - self.c[i]
        if self.L:
            d = d - self.cells * torch.round(d / self.cells).to(torch.int64)
            return (d.abs() <= 1).all(-1)
        cj = self.c[j]
        return ((d.abs() <= 1) & (cj >= 0) & (cj < self.cells)).all(-1)


def _pairs(x, R, L):
    """Ordered pairs (i, j) closer than R, i ascending."""
    n, dev = len(x), x.device
    lo = x.amin(0)
    span = (x.amax(0) - lo).max().item() + 1e-6
    m = max(1, int((L if L else span) / R))
    if n <= 3000 or (L and m < 3):
        step = max(1, (1 << 25) // n)
        out = []
        for a in range(0, n, step):
            d = x[a:a + step, None] - x[None]
            if L:
                d = d - L * torch.round(d / L)
            hit = (d.square().sum(-1) < R * R).nonzero()
            hit[:, 0] += a
            out.append(hit[hit[:, 0] != hit[:, 1]])
        p = torch.cat(out)
        return p[:, 0], p[:, 1]
    if L:
        cell = torch.floor((x + L / 2) / (L / m)).to(torch.int64) % m
    else:
        cell = torch.floor((x - lo) / (span / m)).to(torch.int64).clamp(0, m - 1)
    flat = (cell[:, 0] * m + cell[:, 1]) * m + cell[:, 2]
    order = torch.argsort(flat, stable=True)
    count = torch.bincount(flat, minlength=m ** 3)
    start = torch.cumsum(count, 0) - count
    cap = int(count.max())
    off = torch.tensor([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)],
                       device=dev)
    slot = torch.arange(cap, device=dev)
    step = max(1, (1 << 27) // (27 * cap))
    ii, jj = [], []
    for a in range(0, n, step):
        c = cell[a:a + step, None] + off[None]
        ok = torch.ones(c.shape[:2], dtype=torch.bool, device=dev)
        if L:
            c = c % m
        else:
            ok = ((c >= 0) & (c < m)).all(-1)
            c = c.clamp(0, m - 1)
        f = (c[..., 0] * m + c[..., 1]) * m + c[..., 2]
        idx = start[f][..., None] + slot
        ok = ok[..., None] & (slot < count[f][..., None])
        cand = order[torch.where(ok, idx, torch.zeros_like(idx))]
        d = x[a:a + step, None, None] - x[cand]
        if L:
            d = d - L * torch.round(d / L)
        me = torch.arange(a, min(a + step, n), device=dev)[:, None, None]
        hit = (ok & (d.square().sum(-1) < R * R) & (cand != me)).nonzero(as_tuple=True)
        ii.append(hit[0] + a)
        jj.append(cand[hit])
    return torch.cat(ii), torch.cat(jj)


class _Exact:
    """The run of one box in 64 bits: LJ and bond order over the engine's candidates."""

    def __init__(self, pos, vel, L, nmb, table, dt, mb_force=None):
        self.x, self.type = _tens(pos[:, :3]), torch.as_tensor(pos[:, 3].astype(np.int64),
                                                               device=_dev())
        self.v, self.L, self.nmb, self.n = _tens(vel), L, nmb, len(pos)
        self.use_lj = nmb < self.n
        ng = (3.405, 9.960172e-5, 39.948) if table == "argon" else (2.72, 0.391e-4, 20.1797)
        f = lambda *a: torch.tensor([float(F32(t)) for t in a], dtype=torch.float64,  # noqa: E731
                                    device=_dev())
        self.sig, self.eps = f(3.015, 2.835, ng[0]), f(0.328e-4, 0.447e-4, ng[1])
        self.mass = f(14.00674, 15.9994, ng[2])[self.type][:, None]
        # a run's first forces are the bond order's, whatever drives it afterwards
        self.dt, self.mb_force, self.mb_next = float(F32(dt)), _bond_order, mb_force
        self.next = {"lj": 0, "mb": 0}

    def speed(self):
        return float(self.v.square().sum(1).sqrt().max())

    def due(self, t):
        return t in [self.next[k] for k, on in (("lj", self.use_lj), ("mb", self.nmb > 0)) if on]

    def lists(self, t, vmax):
        due = [k for k, on in (("lj", self.use_lj), ("mb", self.nmb > 0))
               if on and (self.next[k] == t or self.L)]
        if self.L:
            self.x = self.x - self.L * torch.floor((self.x + self.L / 2) / self.L)
        for k in due:
            rs, rc = (RS, RC) if k == "lj" else (MB_RS, MB_RC)
            x = self.x if k == "lj" else self.x[:self.nmb]
            xr = self.x  # the walls' box follows the farthest atom of all
            cells = _Cells(xr, rs, self.L)
            i, j = _pairs(x, rs + 0.5 if not self.L or self.L > 2 * rs + 1 else rs, self.L)
            keep = cells.adjacent(i, j)
            if k == "lj":
                keep &= (self.type[i] == 2) | (self.type[j] == 2)
                self.i, self.j = i[keep], j[keep]
                sel = torch.where(self.type[self.i] == 2, self.type[self.j], self.type[self.i])
                self.s2, self.e24 = self.sig[sel].square(), 24 * self.eps[sel]
                if len(torch.unique(sel)) <= 1:
                    self.s2, self.e24 = self.s2[:1], self.e24[:1]
            else:
                self.mi, self.mj, self.mcells = i[keep], j[keep], cells
            move = float((F32(rs) - F32(rc)) * F32(0.5))
            q = move / vmax / self.dt if vmax > 0 else 1e18
            self.next[k] = t + (int(q) if q < 2e9 else 2 ** 31)
        if self.L:
            m = min(self.next[k] for k in due)
            for k in due:
                self.next[k] = m

    def delta(self, i, j):
        d = self.x[i] - self.x[j]
        return d - self.L * torch.round(d / self.L) if self.L else d

    def forces(self):
        f = torch.zeros_like(self.x)
        if self.use_lj:
            rc2 = float(F32(float(F32(RC)) ** 2))
            for a in range(0, len(self.i), 1 << 25):
                i, j = self.i[a:a + (1 << 25)], self.j[a:a + (1 << 25)]
                s2 = self.s2[a:a + (1 << 25)] if len(self.s2) > 1 else self.s2
                e24 = self.e24[a:a + (1 << 25)] if len(self.e24) > 1 else self.e24
                d = self.delta(i, j)
                r2 = d.square().sum(1)
                q = s2 / r2
                q3 = q * q * q
                w = torch.where(r2 < rc2, e24 / s2 * q * q3 * (2 * q3 - 1), torch.zeros_like(r2))
                f.index_add_(0, i, d * w[:, None])
        if self.nmb:
            f[:self.nmb] += self.mb_force(self)
        return f

    def start(self):
        """a = F/m, b = c = 0"""
        self.a = self.forces() / self.mass
        self.mb_force = self.mb_next or self.mb_force
        self.b, self.c = torch.zeros_like(self.a), torch.zeros_like(self.a)

    def step(self):
        dt, g = self.dt, [float(F32(t)) for t in (0.15833333333333333, 0.75, 0.5,
                                                  0.08333333333333333)]
        c1 = dt
        c2 = c1 * dt / 2
        c3 = c2 * dt / 3
        c4 = c3 * dt / 4
        cr, cv, cb, cc = g[0] * c2, g[1] * c2 / c1, g[2] * c2 / c3, g[3] * c2 / c4
        self.x = self.x + c1 * self.v + c2 * self.a + c3 * self.b + c4 * self.c
        self.v = self.v + c1 * self.a + c2 * self.b + c3 * self.c
        self.a = self.a + c1 * self.b + c2 * self.c
        self.b = self.b + c1 * self.c
        self.f = self.forces()
        a = self.f / self.mass
        d = a - self.a
        self.x, self.v, self.a = self.x + cr * d, self.v + cv * d, a
        self.b, self.c = self.b + cb * d, self.c + cc * d


def _run(systems, steps):
    """Positions (with the species) and velocities after `steps` of systems that share the list
    schedule: the fastest atom of all decides."""
    for t in range(steps):
        if t == 0 or any(s.due(t) for s in systems):
            vmax = max(s.speed() for s in systems)
            for s in systems:
                s.lists(t, vmax)
                if t == 0:
                    s.start()
        for s in systems:
            s.step()
    return (torch.cat([torch.cat([s.x, s.type[:, None].double()], 1) for s in systems]),
            torch.cat([s.v for s in systems]))


def _cut(r):
    t = torch.tanh(2.0 * (r - float(F32(1.3))))
    return 0.5 * (1 - t), -(1 - t * t)


def _angle(c):
    D = float(F32(4.0417))
    q = D + c * c
    k = float(F32(1) + F32(25) / F32(4.0417))
    return k - 25 / q, 50 * c / (q * q)


def _table(i, j, n, keep):
    """Padded neighbour table (n, S): index and validity, neighbours in pair order."""
    i, j = i[keep], j[keep]
    count = torch.bincount(i, minlength=n)
    S = max(1, int(count.max()))
    slot = torch.arange(len(i), device=i.device) - (torch.cumsum(count, 0) - count)[i]
    nb = torch.zeros(n, S, dtype=torch.int64, device=i.device)
    nb[i, slot] = j
    ok = torch.arange(S, device=i.device)[None] < count[:, None]
    return nb, ok


def _bond_order(s):
    """Bond-order forces on the many-body atoms: pair terms with the bond order's change along
    r_i, and the third bodies' forces where j is a candidate in the third body's row."""
    n = s.nmb
    f = lambda t: float(F32(t))  # noqa: E731
    d = s.delta(s.mi, s.mj)
    keep = d.square().sum(1) < float(F32(f(MB_RC) ** 2))
    nb, ok = _table(s.mi, s.mj, n, keep)
    S = nb.shape[1]
    out = torch.zeros(n, 3, dtype=torch.float64, device=nb.device)
    third = torch.zeros(n, 3, dtype=torch.float64, device=nb.device)
    step = max(1, (1 << 26) // (S * S))
    for a in range(0, n, step):
        me = torch.arange(a, min(a + step, n), device=nb.device)
        N, K = nb[me], ok[me]
        u = s.delta(me[:, None].expand_as(N), N)
        u = torch.where(K[..., None], u, torch.ones_like(u))
        r = u.square().sum(-1).sqrt()
        u = u / r[..., None]
        ti, tj = s.type[me][:, None], s.type[N]
        pick = lambda x, y, z: torch.where(ti == tj, torch.where(  # noqa: E731
            ti == 0, torch.full_like(r, f(x)), torch.full_like(r, f(y))), torch.full_like(r, f(z)))
        re, de = pick(1.097, 1.2075, 1.15), pick(941.4e-4, 493.55309e-4, 626.734e-4)
        beta, r0 = pick(2.71009, 2.2478, 2.24068), pick(3.72, 3.31, 3.51)
        va = 2 * de * torch.exp(-beta * (r - re))
        dva = beta * va
        vr = de * torch.exp(-2 * beta * (r - re)) + f(7.0e-8) * torch.exp(-10 * beta * (r - re))
        dvr = 2 * beta * vr
        gm, gm2 = F32(0.3), F32(0.09)
        al = 3 * (r - r0)
        ep, gx = torch.exp(al), float(gm) * torch.exp(-al)
        A, B = ep + gx, 3 * (ep - gx)
        k10 = float(F32(10) * (gm - F32(1)))
        v = float(F32(1) + F32(50) * gm + gm2) + k10 * B
        dvdw = -f(1.0e-4) * ((k10 * (9 * A) * A - 2 * B * v) / (A * A * A))
        lam = f(1.33)
        E = torch.exp(lam * (r - re))
        fcm, dfcm = _cut(r)
        j, m = (slice(None), slice(None), None), (slice(None), None, slice(None))
        use = K[j] & K[m] & ~torch.eye(S, dtype=torch.bool, device=nb.device)
        uj, um = u[:, :, None], u[:, None]
        vec = um * r[m][..., None] - uj * r[j][..., None]        # r_j - r_m
        rjm = torch.where(use, vec.square().sum(-1).sqrt(), torch.ones_like(use, dtype=r.dtype))
        fj, dfj = _cut(rjm)
        rij, rim = r[j], r[m]
        ic = (rij * rij + rim * rim - rjm * rjm) / (2 * rij * rim)
        jc = (rij * rij + rjm * rjm - rim * rim) / (2 * rij * rjm)
        gi, pi = _angle(ic)
        gj, pj = _angle(jc)
        fi, dfi, Ej = fcm[m], dfcm[m], E[j]
        z = lambda t: torch.where(use, t, torch.zeros_like(t))  # noqa: E731
        xi, xj = z(fi * gi * Ej).sum(2), z(fj * gj * Ej).sum(2)
        Ai = dfi * gi + fi * pi * (1 / rij - ic / rim)
        Bj = -fj * pj * rim / (rij * rjm)
        ci = fi * (pi * (1 / rim - ic / rij) + gi * lam)
        cj = fj * (pj * (1 / rjm - jc / rij) + gj * lam)
        dxi = (z(Ej * Ai)[..., None] * um).sum(2) + z(Ej * ci).sum(2)[..., None] * u
        dxj = (z(Ej * Bj)[..., None] * um).sum(2) + z(Ej * cj).sum(2)[..., None] * u
        pbi, pbj = 1 / (1 + xi) ** 2, 1 / (1 + xj) ** 2
        bo = 0.5 * (1 / (1 + xi) + 1 / (1 + xj))
        db = 0.5 * (pbi[..., None] * dxi + pbj[..., None] * dxj)
        fij = dvr - bo * dva + dvdw
        out[me] = torch.where(K[..., None], fij[..., None] * u - va[..., None] * db,
                              torch.zeros_like(u)).sum(1)
        wi, wj = (0.25 * va * E * pbi)[j], (0.25 * va * E * pbj)[j]
        seen = s.mcells.adjacent(N[m].expand_as(use), N[j].expand_as(use))
        y = lambda t: torch.where(use & seen, t, torch.zeros_like(t))  # noqa: E731
        ck = y(wi * Ai + wj * Bj)
        cjm = y(-wi * fi * pi * rjm / (rij * rim) +
                wj * (dfj * gj + fj * pj * (1 / rij - jc / rjm)))
        fm = ck.sum(1)[..., None] * u + (cjm / rjm)[..., None].mul(vec).sum(1)
        third.index_add_(0, N[K], fm[K])
    return out + third


def _descriptor_forces(w_of):
    """Forces -sum_i w_i . dG_i/dr_j of the symmetry functions within 3 angstrom."""
    rc = 3.0
    dd = (rc - 0.8) / 15.0
    k = torch.arange(16, device=_dev())
    rk, eta = 0.8 + dd * k.double(), 0.5 / (dd * dd)
    zeta = torch.tensor([1.0, 2.0, 4.0, 16.0], dtype=torch.float64, device=_dev())[k % 4]
    lam = torch.where((k // 4) % 2 == 1, -1.0, 1.0).double()
    ea = torch.tensor([0.02, 0.25], dtype=torch.float64, device=_dev())[k // 8]
    pref = 2.0 ** (1.0 - zeta)

    def forces(s):
        n = s.nmb
        d = s.delta(s.mi, s.mj)
        nb, ok = _table(s.mi, s.mj, n, d.square().sum(1) < rc * rc)
        S = nb.shape[1]
        grad = torch.zeros(n, 3, dtype=torch.float64, device=nb.device)
        a, b = torch.triu_indices(S, S, 1, device=nb.device)
        step = max(1, (1 << 25) // (16 * len(a) + 1))
        for c in range(0, n, step):
            me = torch.arange(c, min(c + step, n), device=nb.device)
            N, K = nb[me], ok[me]
            u = -s.delta(me[:, None].expand_as(N), N)
            u = torch.where(K[..., None], u, torch.ones_like(u)).requires_grad_()
            r = u.square().sum(-1).sqrt()
            fc = torch.where(K, 0.5 * (torch.cos(math.pi * r / rc) + 1), torch.zeros_like(r))
            g2 = (torch.exp(-eta * (r[..., None] - rk) ** 2) * fc[..., None]).sum(1)
            cs = (u[:, a] * u[:, b]).sum(-1) / (r[:, a] * r[:, b])
            q, ff = r[:, a] ** 2 + r[:, b] ** 2, fc[:, a] * fc[:, b]
            base = torch.clamp(1 + lam * cs[..., None], min=0.0)
            g4 = (pref * base ** zeta * torch.exp(-ea * q[..., None]) * ff[..., None]).sum(1)
            G = torch.cat([g2, g4], 1)
            gu, = torch.autograd.grad((G * w_of(G.detach())).sum(), u)
            gu = torch.where(K[..., None], gu, torch.zeros_like(gu))
            grad.index_add_(0, N[K], gu[K])
            grad[me] -= gu.sum(1)
        return -grad

    return forces


def _head_weights(case, seed):
    """G -> w of the seeded head, in 64 bits."""
    h, p, o, t = case["hidden"], _tens(_head(case["hidden"], seed)), 0, []
    for shape in ((h, 32), (h,), (h, h), (h,), (32, h), (32,)):
        k = math.prod(shape)
        t.append(p[o:o + k].reshape(shape))
        o += k
    istd = float(F32(DESC_ISTD))

    def w(G):
        x = (G - DESC_MEAN) * istd
        y = torch.tanh(torch.tanh(x @ t[0].T + t[1]) @ t[2].T + t[3]) @ t[4].T + t[5]
        return y * HEAD_SCALE * istd

    return w


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        # Adam steps on tensor-core gradients: each weight moves by the learning rate times a
        # ratio of running means of those gradients, which has no 64-bit value of its own
        return None
    if kind == "batch":
        pos, vel, natoms, boxes = _ensemble(case, seed)
        systems, a = [], 0
        for k, L in zip(natoms, boxes):
            systems.append(_Exact(pos[a:a + k], vel[a:a + k], float(L), 0, "argon", case["dt"]))
            a += k
        p, v = _run(systems, case["steps"])
        return {"pos": p, "vel": v}
    pos, vel, L, nmb, table = _inputs(case, seed)
    if kind == "calls":
        s = _Exact(pos, vel, 0.0, 0, table, 2.0)
        p, v = _run([s], 1)
        # a = F/m; b and c hold the correction alone, a difference of nearly equal forces
        return {"rows": None, "force": s.f, "pos": p, "vel": v, "acc": s.a, "b": None, "c": None,
                "thermo": None}
    mb = _descriptor_forces(_head_weights(case, seed)) if kind == "surrogate" else None
    periodic = case.get("periodic", kind in ("lj32", "bo32", "surrogate"))
    s = _Exact(pos, vel, L if periodic else 0.0, nmb, table, case["dt"], mb)
    p, v = _run([s], case["steps"])
    out = {"pos": p, "vel": v}
    if case.get("records"):
        out["records"] = None
    return out
