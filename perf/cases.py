"""The work a molecular-dynamics program has this framework do, as cases to time.

Systems are chains in flexible water at about 100 atoms/nm^3, as
nexusmd_gb300.synthetic makes them: a unit box of one chain and its waters,
repeated along each axis (the repeats shifted against one another by the
seed's jitter), with a few waters left out where a case wants an odd atom
count.  The sizes are those of the benchmark's configurations (2,700 atoms on
a 32^3 PME grid, 23,800 on 64^3, 94,100 on 100^3, 473,400 on 180^3 at a 1.2
nm cutoff, and a batch of 32 systems of 2,000 to 25,000 atoms), and odd ones
between them in boxes of unequal edges.  The seed shifts the whole system
through its periodic box, exchanges and mirrors its axes, displaces every
atom a little and draws the velocities, so another seed is another input.

Kinds of work:
  forces  new positions into a context that is kept, forces and energies out
          (a minimiser, a Monte Carlo move, labels for a fitted potential);
  steps   new positions and velocities into a context that is kept, a block of
          leapfrog steps, the state after them and the last step's energies
          out (replicas or windows that exchange their states between blocks);
  frames  the same, with every step's positions and energies read back while
          the next step runs;
  job     a context made from host arrays, velocities set, a few steps with
          every frame read back, the context given back (a short job);
  pme     the reciprocal-space entry point on the caller's device buffers.

Values of the mixed-precision engine are handed on as FP32, the width of its
force arithmetic and of the trajectory and training files that keep them;
those of the FP64 engine as FP64.
"""
from __future__ import annotations

import ctypes
import dataclasses
import functools
import math
import random

import numpy as np
import torch

from nexusmd_gb300 import engine as nxe
from nexusmd_gb300 import synthetic as syn

DT = 0.0005  # ps
KE = 138.93545764446428693393  # kJ nm / (mol e^2)
TERMS = ("bond", "angle", "torsion", "recip", "self", "coulomb", "vdw", "exclusion", "kinetic", "potential",
         "exception")


# ------------------------------------------------------------------ cases

def _case(kind, precision, unit, tiles, grid, cutoff=1.0, tol=5e-4, drop=0, steps=0, systems=1, switch=0.0, name=None):
    c = {} if name is None else {"name": name}
    c.update(kind=kind, precision=precision, unit=unit, mx=tiles[0], my=tiles[1], mz=tiles[2], gx=grid[0], gy=grid[1],
             gz=grid[2], cutoff=cutoff, tol=tol, drop=drop, steps=steps, systems=systems, switch=switch)
    return c


def listed():
    return [
        # the smallest system of the configurations, in the reference's own
        # precision and without exceptions: one energy-and-force call
        _case("forces", "fp64", 2700, (1, 1, 1), (32, 32, 32), name="forces_fp64_2700"),
        # the same call of the mixed engine: what is left is latency
        _case("forces", "mixed", 2700, (1, 1, 1), (32, 32, 32), name="forces_mixed_2700"),
        # a small system stepped: a hundred launches of the step
        _case("steps", "mixed", 2700, (1, 1, 1), (32, 32, 32), steps=100, name="steps_mixed_2700"),
        # the second configuration in both precisions
        _case("steps", "fp64", 2975, (2, 2, 2), (64, 64, 64), steps=3, name="steps_fp64_24k"),
        _case("steps", "mixed", 2975, (2, 2, 2), (64, 64, 64), steps=50, name="steps_mixed_24k"),
        # an odd size in a box of unequal edges on a grid with odd axes, with
        # the Lennard-Jones switching function on, as many exported systems have it
        _case("forces", "mixed", 3102, (2, 3, 4), (64, 96, 125), drop=7, switch=0.9, name="forces_mixed_74k_switch"),
        # the benchmark's headline configuration: 20 steps as it times them,
        # the same with every frame read back, and end to end
        _case("steps", "mixed", 3486, (3, 3, 3), (100, 100, 100), steps=20, name="steps_mixed_94k"),
        _case("frames", "mixed", 3486, (3, 3, 3), (100, 100, 100), steps=10, name="frames_mixed_94k"),
        _case("job", "mixed", 3486, (3, 3, 3), (100, 100, 100), steps=20, name="job_mixed_94k"),
        # many uneven systems in one context (lambda windows)
        _case("steps", "mixed", 0, (1, 1, 1), (0, 0, 0), steps=8, systems=32, name="batch32_mixed"),
        # the largest configuration: long cutoff, tight Ewald tolerance
        _case("steps", "mixed", 3786, (5, 5, 5), (180, 180, 180), cutoff=1.2, tol=1e-5, steps=6,
              name="steps_mixed_473k"),
        # reciprocal space alone, on another program's device buffers
        _case("pme", "mixed", 2975, (2, 2, 2), (64, 64, 64), name="pme_24k"),
    ]


# unit boxes that the generator is known to fill
UNITS = (2050, 2250, 2500, 2700, 2975, 3102, 3250, 3486, 3786)


def draw(rng: random.Random):
    kind = rng.choice(["forces", "steps", "steps", "frames", "job", "pme", "forces", "steps"])
    precision = "fp64" if kind in ("forces", "steps") and rng.random() < 0.3 else "mixed"
    unit = rng.choice(UNITS)
    if kind == "steps" and precision == "mixed" and rng.random() < 0.3:
        return _case("steps", "mixed", 0, (1, 1, 1), (0, 0, 0), drop=rng.randrange(0, 20), steps=rng.randrange(2, 9),
                     systems=rng.randrange(2, 33))
    # tiles per axis: log-uniform in the number of unit boxes
    most = {"fp64": 8, "mixed": 64}[precision] if kind != "pme" else 8
    target = math.exp(rng.uniform(0.0, math.log(most)))
    tiles = [1, 1, 1]
    while tiles[0] * tiles[1] * tiles[2] < target * 0.8:
        tiles[rng.randrange(3)] += 1
        if max(tiles) > 4:
            tiles = sorted(tiles)
            tiles[2] = 4
            tiles[0] += 1
    if kind == "pme":
        tiles = [min(t, 2) for t in tiles]
    edge = _edge(unit)
    grid = []
    for t in tiles:
        g = syn.smooth_grid(max(8, int(math.ceil(t * edge * rng.uniform(9.0, 11.0)))))
        grid.append(min(g, 64) if kind == "pme" else g)
    n = unit * tiles[0] * tiles[1] * tiles[2]
    steps = 0
    if kind in ("steps", "frames", "job"):
        steps = rng.randrange(1, 4) if precision == "fp64" else rng.randrange(2, max(3, min(60, 1200000 // n)))
        steps = min(steps, 20) if kind != "steps" else steps
    switch = 0.9 if kind == "forces" and rng.random() < 0.25 else 0.0
    cutoff = 1.0 if kind == "pme" or switch else rng.choice([0.9, 1.0, 1.0])
    return _case(kind, precision, unit, tiles, grid, cutoff=cutoff, tol=rng.choice([5e-4, 1e-4]),
                 drop=rng.randrange(0, 40), steps=steps, switch=switch)


# ----------------------------------------------------------------- inputs

def _edge(unit):
    return (unit / 100.0) ** (1.0 / 3.0)


@functools.lru_cache(maxsize=None)
def _unit(unit):
    residues = int(round(0.08 * unit / 8))
    waters = int(round((unit - 8 * residues) / 3))
    return syn.make_system(1, residues, waters, _edge(unit), 7000 + unit)


@functools.lru_cache(maxsize=4)
def _tiled(unit, tiles, drop, charge_scale):
    """The unit box repeated, without `drop` of its waters; chain charges scaled."""
    u = _unit(unit)
    m = tiles[0] * tiles[1] * tiles[2]
    shift = np.stack(np.meshgrid(*[np.arange(t) for t in tiles], indexing="ij"), -1).reshape(-1, 3) * _edge(unit)
    chain = len(u.torsions) + 3
    q = u.charge.copy()
    q[:chain] *= charge_scale

    def atoms(a):
        return np.tile(a, m)

    def idx(a):
        return (a[None] + (u.n * np.arange(m))[:, None, None]).reshape(-1, a.shape[1]).astype(np.int32)

    def prm(a):
        return np.tile(a, (m,) + (1,) * (a.ndim - 1))

    s = syn.System(pos=(u.pos[None] + shift[:, None]).reshape(-1, 3), mass=atoms(u.mass), charge=atoms(q),
                   sigma=atoms(u.sigma), epsilon=atoms(u.epsilon), bonds=idx(u.bonds), bond_prm=prm(u.bond_prm),
                   angles=idx(u.angles), angle_prm=prm(u.angle_prm), torsions=idx(u.torsions),
                   torsion_prm=prm(u.torsion_prm), torsion_n=prm(u.torsion_n), box=_edge(unit) * np.array(tiles, float))
    if drop:
        keep = np.ones(s.n, bool)
        waters = (u.n - chain) // 3
        pick = np.random.default_rng(unit + drop).choice(waters, min(drop, waters // 8), replace=False)
        o = (np.arange(len(pick)) % m) * u.n + chain + 3 * pick
        keep[o] = keep[o + 1] = keep[o + 2] = False
        s = syn.subset(s, np.nonzero(keep)[0])
    return s


def _batch_shapes(case):
    """(unit, tiles, lambda) of each system of a batch: sizes log-uniform in 2,000 to 25,000."""
    r = random.Random(41 * case["systems"] + case["drop"])
    out = []
    for k in range(case["systems"]):
        n = math.exp(r.uniform(math.log(2000), math.log(25000)))
        tiles = (1, 1, 1) if n < 3900 else ((1, 1, 2) if n < 7500 else ((1, 2, 2) if n < 15000 else (2, 2, 2)))
        per = n / (tiles[0] * tiles[1] * tiles[2])
        unit = min(UNITS, key=lambda x: abs(x - per))
        out.append((unit, tiles, k / max(1, case["systems"] - 1)))
    return out


def _inputs(case, seed):
    """[(system, velocities)] of a case."""
    rng = np.random.default_rng(seed)
    if case["systems"] > 1:
        shapes = _batch_shapes(case)
    else:
        shapes = [(case["unit"], (case["mx"], case["my"], case["mz"]), 1.0)]
    out = []
    for unit, tiles, lam in shapes:
        s = _tiled(unit, tiles, case["drop"] if case["systems"] == 1 else 0, lam)
        # one periodic shift, an exchange of equal axes, mirror images, and a
        # displacement of each atom
        pos = s.pos + rng.uniform(0.0, 1.0, 3) * s.box
        for a, b in ((0, 1), (1, 2), (0, 2)):
            if tiles[a] == tiles[b] and rng.integers(2):
                pos[:, [a, b]] = pos[:, [b, a]]
        pos *= np.where(rng.integers(2, size=3), 1.0, -1.0)
        pos += rng.uniform(-0.0008, 0.0008, pos.shape)
        pos -= s.box * np.floor(pos / s.box)
        grid = (case["gx"], case["gy"], case["gz"])
        if case["systems"] > 1:
            grid = tuple(syn.smooth_grid(int(math.ceil(e / 0.1))) for e in s.box)
        s = dataclasses.replace(s, pos=np.ascontiguousarray(pos), cutoff=case["cutoff"], ewald_tol=case["tol"],
                                grid=grid)
        if case["precision"] == "mixed":
            s = syn.with_exceptions(s)
        v = rng.normal(size=pos.shape) * np.sqrt(0.0083144626 * 300.0 / s.mass)[:, None]
        v -= (v * s.mass[:, None]).sum(0) / s.mass.sum()
        out.append((s, v))
    return out


def _alpha(case):
    return math.sqrt(-math.log(2.0 * case["tol"])) / case["cutoff"]


class _State:
    """What a program holds: host arrays and a context, or device buffers."""


def _engine(case, systems):
    mixed = case["precision"] == "mixed"
    return nxe.Engine(systems, precision=nxe.PRECISION_MIXED if mixed else nxe.PRECISION_FP64, box="explicit",
                      exceptions=mixed, use_switch=1 if case["switch"] else 0, switch_dist=case["switch"])


def prepare(case, seed):
    made = _inputs(case, seed)
    st = _State()
    st.case = case
    st.systems = [s for s, _ in made]
    st.x = np.concatenate([s.pos for s in st.systems])
    st.v = np.concatenate([v for _, v in made])
    st.out = np.float32 if case["precision"] == "mixed" else np.float64
    if case["kind"] == "pme":
        s = st.systems[0]
        st.lib = nxe.load_library()
        f = st.lib.nxm_pme_reciprocal_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p,
                      ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        f.restype = ctypes.c_int
        st.xyz = torch.tensor(s.pos, dtype=torch.float64, device="cuda")
        st.q = torch.tensor(s.charge, dtype=torch.float64, device="cuda")
        st.lb = (ctypes.c_double * 3)(0.0, 0.0, 0.0)
        st.ub = (ctypes.c_double * 3)(*s.box.tolist())
        st.grid = (ctypes.c_int32 * 3)(*s.grid)
        st.force = torch.empty((s.n, 3), dtype=torch.float64, device="cuda")
        st.energy = torch.empty(1, dtype=torch.float64, device="cuda")
    elif case["kind"] != "job":
        st.engine = _engine(case, st.systems)
    return st


# -------------------------------------------------------------------- run

def _energies(st, one):
    return np.array([one[t] for t in TERMS], st.out)


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "pme":
        stream = torch.cuda.current_stream().cuda_stream
        rc = st.lib.nxm_pme_reciprocal_noalloc(st.xyz.data_ptr(), st.q.data_ptr(), st.xyz.shape[0], st.lb, st.ub, st.grid,
                                               _alpha(case), st.force.data_ptr(), st.energy.data_ptr(), stream)
        if rc != 0:
            raise RuntimeError(st.lib.nxm_last_error().decode())
        return {"force": st.force.float(), "energy": st.energy.float()}
    if kind == "forces":
        st.engine.set_positions(st.x)
        f = st.engine.compute_forces()
        return {"force": f.astype(st.out, copy=False), "energy": _energies(st, st.engine.energies())}
    if kind == "steps":
        e = st.engine
        e.set_positions(st.x)
        e.set_velocities(st.v)
        e.step(case["steps"], DT)
        x, v = e.state()
        return {"x": x.astype(st.out, copy=False), "v": v.astype(st.out, copy=False),
                "energy": np.stack([_energies(st, e.energies(k)) for k in range(len(st.systems))])}
    # frames and job: every step's frame, the copy of one beside the next step
    e = st.engine if kind == "frames" else _engine(case, st.systems)
    if kind == "frames":
        e.set_positions(st.x)
    e.set_velocities(st.v)
    xs, es = [], []

    def take():
        x, en = e.frame_wait(copy=False)
        xs.append(x.astype(st.out))
        es.append(_energies(st, en))

    e.step_async(1, DT)
    for _ in range(case["steps"] - 1):
        e.step_async(1, DT)
        take()
    take()
    if kind == "job":
        e.close()
    return {"x": xs, "energy": np.stack(es)}


# ------------------------------------------------------------------- work

def work(case):
    """Bytes and operations of one pass, from the sizes: per evaluation 60
    operations per pair within the cutoff, 38 per grid point of a spread and
    gather of 125 points each and 5 N log2 N each way of the half-spectrum
    transform per grid point; per evaluation and atom the positions, charges,
    forces and state read and written once (152 bytes in the step), the grid
    once each way through the transform; and the host's arrays that come and go."""
    sizes = _batch_shapes(case) if case["systems"] > 1 else [(case["unit"], (case["mx"], case["my"], case["mz"]), 1.0)]
    flops = nbytes = 0.0
    evals = max(1, case["steps"])
    for unit, tiles, _ in sizes:
        m = tiles[0] * tiles[1] * tiles[2]
        n = unit * m - (3 * case["drop"] if case["systems"] == 1 else 0)
        edge = [_edge(unit) * t for t in tiles]
        grid = [syn.smooth_grid(int(math.ceil(e / 0.1))) for e in edge] if case["systems"] > 1 else \
            [case["gx"], case["gy"], case["gz"]]
        pts = grid[0] * grid[1] * grid[2]
        word = 4.0 if case["precision"] == "mixed" else 8.0
        fft = 5.0 * pts * math.log2(pts)
        spread = n * (125 * 2 + 125 * 6 + 60)
        if case["kind"] == "pme":
            return {"bytes": n * (32.0 + 24.0) + 8.0 + 4 * word * pts, "flops": fft + spread}
        pairs = n * 100.0 * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3 / 2
        flops += evals * (60.0 * pairs + fft + spread + n * 60.0)
        nbytes += evals * (n * 152.0 + 4 * word * pts + n * 2.0 * pairs / n)
        nbytes += n * 24.0 * {"forces": 2, "steps": 4}.get(case["kind"], 3)
        if case["kind"] in ("frames", "job"):
            nbytes += (case["steps"] - 1) * n * 24.0
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ exact

def _spline(fr):
    """Order-5 B-spline weights at fractions fr [n]: w[k] = M5(fr + 4 - k), and their derivatives."""
    def up(w, n):  # M_n(u) from M_(n-1), at u = fr + n - 1 - k for k = 0..n-1
        out = []
        for k in range(n):
            u = fr + (n - 1 - k)
            left = w[k - 1] if k > 0 else 0.0       # M_(n-1)(u)
            right = w[k] if k < n - 1 else 0.0      # M_(n-1)(u - 1)
            out.append((u * left + (n - u) * right) / (n - 1))
        return out

    w = [1 - fr, fr]
    for n in (3, 4):
        w = up(w, n)
    d = [-w[0], w[0] - w[1], w[1] - w[2], w[2] - w[3], w[3]]
    return torch.stack(up(w, 5), 1), torch.stack(d, 1)


class _Exact:
    """Forces and energies of one system in 64 bits, from the formulas."""

    def __init__(self, s, case, device):
        self.case, self.dev = case, device
        t = lambda a, dt=torch.float64: torch.tensor(np.asarray(a), dtype=dt, device=device)  # noqa: E731
        self.n, self.box, self.alpha = s.n, t(s.box), _alpha(case)
        self.q, self.mass, self.sig, self.eps = t(s.charge), t(s.mass), t(s.sigma), t(s.epsilon)
        self.terms = [(t(s.bonds, torch.int64), t(s.bond_prm)), (t(s.angles, torch.int64), t(s.angle_prm)),
                      (t(s.torsions, torch.int64), t(s.torsion_prm))]
        self.per = t(s.torsion_n)
        # within three bonds: the ends of bonds, angles and torsions (no rings)
        ex = [np.asarray(s.bonds), np.asarray(s.angles)[:, [0, 2]], np.asarray(s.torsions)[:, [0, 3]]]
        # a triangle-free three-site molecule has its far pair in the angle list
        ex = np.unique(np.sort(np.concatenate(ex), axis=1), axis=0)
        self.ex = t(ex, torch.int64)
        self.exkey = torch.sort(self.ex[:, 0] * self.n + self.ex[:, 1])[0]
        self.xc = None
        if s.exc_idx is not None and len(s.exc_idx):
            self.xc = (t(s.exc_idx, torch.int64), t(s.exc_prm))
        self.K = tuple(int(k) for k in s.grid)
        self.influence()

    def influence(self):
        K, V = self.K, float(torch.prod(self.box))
        mods, ms = [], []
        m5 = [1 / 24, 11 / 24, 11 / 24, 1 / 24]
        for d in range(3):
            k = torch.arange(K[d], dtype=torch.float64, device=self.dev)
            b = sum(c * torch.exp(2j * math.pi * k * (j + 1) / K[d]) for j, c in enumerate(m5)).abs() ** 2
            for i in (b < 1e-7).nonzero().flatten().tolist():
                b[i] = (b[i - 1] + b[(i + 1) % K[d]]) / 2
            mods.append(b)
            ms.append(torch.where(k < (K[d] + 1) // 2, k, k - K[d]) / self.box[d])
        h = K[2] // 2 + 1
        m2 = ms[0][:, None, None] ** 2 + ms[1][None, :, None] ** 2 + ms[2][None, None, :h] ** 2
        den = math.pi * V * m2 * mods[0][:, None, None] * mods[1][None, :, None] * mods[2][None, None, :h]
        den[0, 0, 0] = 1.0
        self.et = KE * torch.exp(-math.pi ** 2 * m2 / self.alpha ** 2) / den
        self.et[0, 0, 0] = 0.0

    def pairs(self, x, reach):
        """Pairs i, j (each once, not excluded) within `reach`: windows of the atoms sorted along x."""
        order = torch.argsort(x[:, 0])
        xs = x[order].float()
        box = self.box.float()
        keys = xs[:, 0].contiguous()
        L = float(box[0])
        got = []
        step = 1024
        for a in range(0, self.n, step):
            b = min(self.n, a + step)
            lo, hi = float(keys[a]) - reach - 1e-4, float(keys[b - 1]) + reach + 1e-4
            spans = [(lo, hi)]
            if hi - lo >= L:
                spans = [(-1.0, L + 1.0)]
            else:
                spans += [(lo + L, L + 1.0)] if lo < 0 else []
                spans += [(-1.0, hi - L)] if hi > L else []
            for s0, s1 in spans:
                c0, c1 = torch.searchsorted(keys, torch.tensor([s0, s1], device=self.dev)).tolist()
                if c1 <= c0:
                    continue
                r2 = 0.0
                for d in range(3):
                    dd = (xs[a:b, d, None] - xs[None, c0:c1, d]).abs()
                    dd = torch.minimum(dd, box[d] - dd)
                    r2 = r2 + dd * dd
                i, j = (r2 < (reach + 1e-4) ** 2).nonzero(as_tuple=True)
                i, j = order[a + i], order[c0 + j]
                keep = i < j
                got.append(torch.stack([i[keep], j[keep]]))
        p = torch.cat(got, 1)
        key = p[0] * self.n + p[1]
        at = torch.searchsorted(self.exkey, key).clamp(max=max(0, len(self.exkey) - 1))
        return p[:, self.exkey[at] != key] if len(self.exkey) else p

    def image(self, d):
        return d - self.box * torch.round(d / self.box)

    def recip(self, x):
        K = self.K
        idx, w, dw = [], [], []
        for d in range(3):
            u = x[:, d] / self.box[d]
            u = (u - torch.floor(u)) * K[d]
            i = torch.floor(u)
            a, b = _spline(u - i)
            idx.append((i.long()[:, None] + torch.arange(5, device=self.dev)) % K[d])
            w.append(a)
            dw.append(b)
        flat = ((idx[0][:, :, None, None] * K[1] + idx[1][:, None, :, None]) * K[2] + idx[2][:, None, None, :]).reshape(self.n, -1)
        prod = lambda a, b, c: (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(len(a), -1)  # noqa: E731
        g = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64, device=self.dev)
        g.index_add_(0, flat.reshape(-1), (prod(*w) * self.q[:, None]).reshape(-1))
        S = torch.fft.rfftn(g.reshape(K))
        wt = torch.full((S.shape[2],), 2.0, dtype=torch.float64, device=self.dev)
        wt[0] = 1.0
        if K[2] % 2 == 0:
            wt[-1] = 1.0
        e = 0.5 * (self.et * (S.real ** 2 + S.imag ** 2) * wt).sum()
        phi = torch.fft.irfftn(S * self.et, s=K, norm="forward").reshape(-1)[flat]
        f = [-(self.q * (K[d] / self.box[d])) * (phi * prod(*[dw[k] if k == d else w[k] for k in range(3)])).sum(1)
             for d in range(3)]
        return float(e), torch.stack(f, 1)

    def bonded(self, x):
        x = x.detach().requires_grad_(True)
        e = []
        (b, bp), (a, ap), (t, tp) = self.terms
        r = self.image(x[b[:, 1]] - x[b[:, 0]]).norm(dim=1)
        e.append((0.5 * bp[:, 1] * (r - bp[:, 0]) ** 2).sum())
        v0, v1 = self.image(x[a[:, 0]] - x[a[:, 1]]), self.image(x[a[:, 2]] - x[a[:, 1]])
        th = torch.atan2(torch.linalg.cross(v0, v1).norm(dim=1), (v0 * v1).sum(1))
        e.append((0.5 * ap[:, 1] * (th - ap[:, 0]) ** 2).sum())
        u0, u1, u2 = (self.image(x[t[:, k]] - x[t[:, m]]) for k, m in ((0, 1), (2, 1), (2, 3)))
        c0, c1 = torch.linalg.cross(u0, u1), torch.linalg.cross(u1, u2)
        phi = torch.atan2(u1.norm(dim=1) * (u0 * c1).sum(1), (c0 * c1).sum(1))
        e.append((tp[:, 0] * (1 + torch.cos(self.per * phi - tp[:, 1]))).sum())
        f = -torch.autograd.grad(sum(e), x)[0]
        return [float(v.detach()) for v in e], f

    def evaluate(self, x, pairs):
        """(forces, {term: energy}) at x; `pairs` holds every pair within the cutoff."""
        en = dict.fromkeys(TERMS, 0.0)
        (en["bond"], en["angle"], en["torsion"]), f = self.bonded(x)
        en["recip"], fr = self.recip(x)
        f = f + fr
        en["self"] = -KE * self.alpha / math.sqrt(math.pi) * float((self.q ** 2).sum())
        rc, sw = self.case["cutoff"], self.case["switch"]
        al = self.alpha
        for a in range(0, pairs.shape[1], 1 << 24):
            i, j = pairs[:, a:a + (1 << 24)]
            d = self.image(x[i] - x[j])
            r2 = (d * d).sum(1)
            near = r2 < rc * rc
            i, j, d, r2 = i[near], j[near], d[near], r2[near]
            r = torch.sqrt(r2)
            qq = KE * self.q[i] * self.q[j]
            ec = qq * torch.erfc(al * r) / r
            g = (ec + qq * 2 * al / math.sqrt(math.pi) * torch.exp(-(al * r) ** 2)) / r2
            s6 = ((0.5 * (self.sig[i] + self.sig[j])) ** 2 / r2) ** 3
            e4 = 4 * torch.sqrt(self.eps[i] * self.eps[j])
            ev, gv = e4 * (s6 * s6 - s6), e4 * (12 * s6 * s6 - 6 * s6) / r2
            if sw:
                u = ((r - sw) / (rc - sw)).clamp(min=0.0)
                S = 1 - 10 * u ** 3 + 15 * u ** 4 - 6 * u ** 5
                dS = (-30 * u ** 2 + 60 * u ** 3 - 30 * u ** 4) / (rc - sw)
                gv = gv * S - ev * dS / r
                ev = ev * S
            en["coulomb"] += float(ec.sum())
            en["vdw"] += float(ev.sum())
            fp = d * (g + gv)[:, None]
            f.index_add_(0, i, fp)
            f.index_add_(0, j, -fp)
        i, j = self.ex[:, 0], self.ex[:, 1]
        d = self.image(x[i] - x[j])
        r = d.norm(dim=1)
        qq = KE * self.q[i] * self.q[j]
        ee = qq * torch.erf(al * r) / r
        fp = -d * ((ee - qq * 2 * al / math.sqrt(math.pi) * torch.exp(-(al * r) ** 2)) / r ** 2)[:, None]
        en["exclusion"] = float(ee.sum())
        f.index_add_(0, i, fp)
        f.index_add_(0, j, -fp)
        if self.xc is not None:
            (p, prm) = self.xc
            i, j = p[:, 0], p[:, 1]
            d = self.image(x[i] - x[j])
            r2 = (d * d).sum(1)
            s6 = (prm[:, 1] ** 2 / r2) ** 3
            c = KE * prm[:, 0] / torch.sqrt(r2)
            en["exception"] = float((c + 4 * prm[:, 2] * (s6 * s6 - s6)).sum())
            fp = d * ((c + 4 * prm[:, 2] * (12 * s6 * s6 - 6 * s6)) / r2)[:, None]
            f.index_add_(0, i, fp)
            f.index_add_(0, j, -fp)
        en["potential"] = sum(en[k] for k in TERMS if k not in ("kinetic", "potential", "exclusion")) - en["exclusion"]
        return f, en

    def steps(self, x, v, count):
        """Each of `count` leapfrog steps: the positions and energies of its force evaluation, and the state after it."""
        reach = self.case["cutoff"] + 0.15
        start, pairs = x.clone(), self.pairs(x, reach)
        for k in range(count):
            if float(self.image(x - start).norm(dim=1).max()) > 0.07:
                start, pairs = x.clone(), self.pairs(x, reach)
            f, en = self.evaluate(x, pairs)
            half = v + f / self.mass[:, None] * (0.5 * DT)
            en["kinetic"] = float((0.5 * self.mass * (half * half).sum(1)).sum())
            at = x
            v = v + f / self.mass[:, None] * DT
            x = x + v * DT
            x = x + self.box * ((x < 0).double() - (x > self.box).double())
            yield at, np.array([en[t] for t in TERMS]), x, v


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    xs, vs, es = [], [], []
    for s, v in _inputs(case, seed):
        E = _Exact(s, case, device)
        x = torch.tensor(s.pos, dtype=torch.float64, device=device)
        if kind == "pme":
            e, f = E.recip(x)
            return {"force": f.cpu(), "energy": torch.tensor([e], dtype=torch.float64)}
        if kind == "forces":
            f, en = E.evaluate(x, E.pairs(x, case["cutoff"]))
            return {"force": f.cpu().numpy(), "energy": np.array([en[t] for t in TERMS])}
        got = list(E.steps(x, torch.tensor(v, dtype=torch.float64, device=device), case["steps"]))
        if kind != "steps":
            return {"x": [g[0].cpu().numpy() for g in got], "energy": np.stack([g[1] for g in got])}
        xs.append(got[-1][2].cpu().numpy())
        vs.append(got[-1][3].cpu().numpy())
        es.append(got[-1][1])
    return {"x": np.concatenate(xs), "v": np.concatenate(vs), "energy": np.stack(es)}
