"""The work that users of the Lennard-Jones library have it do, as timed cases.

`listed()` gives the cases, `draw(rng)` more of the same ranges. `prepare`
builds what a program holds before the call (a simulation or a batch with its
read-back buffers), `run` makes one pass through the Python mirror's public
calls and returns what such a program reads, `exact` the same in 64 bits from
plain torch and numpy (velocity Verlet, BAOAB Langevin, Nose-Hoover, eHEX and
the Irving-Kirkwood profile restated there).

Sizes come from the repository's own workloads: the 1000-atom box, the 15,600
and 16,000-atom slabs, the 256,000-atom liquid, the rho 0.4 fluid of 32,768 to
1,048,576 atoms, 512 uneven replicas, the heat-current box, the heat-exchange
box of the conductivity tests, and a packed bed of grains.
"""

import math
import os
import random  # noqa: F401  (draw() takes a random.Random)
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "virial-engine_b200"))

import virial_lj as vl  # noqa: E402

SKIN = 0.3


# ---- the cases ----

def listed():
    return [
        # A small liquid at constant energy, the reference's test box: short
        # bursts of steps between read-outs, bound by launches and latency.
        dict(name="small_1000", kind="box", n=1000, rho=0.8442, aspect=1.0, T=0.72, thermostat="none",
             shifted=False, cutoff=2.5, dt=0.005, steps=20),
        # One frame of an interactive run: a few steps, then a measurement and
        # the particles for drawing.
        dict(name="frame_32768", kind="box", n=32768, rho=0.4, aspect=1.0, T=1.0, thermostat="none",
             shifted=True, cutoff=2.5, dt=0.004, steps=4),
        # The canonical ensemble by Nose-Hoover on a 15,600-molecule liquid
        # slab (the coexistence runs' equilibration).
        dict(name="nose_hoover_15600", kind="box", n=15600, rho=0.26, aspect=7.5, slab=0.366, T=0.7,
             thermostat="nose_hoover", shifted=True, cutoff=2.5, dt=0.005, steps=40),
        # Liquid-vapour coexistence: a 300-bin profile sample every 20 steps.
        dict(name="slab_profile_16000", kind="profile", n=16000, rho=16000 / 60000.0, aspect=7.5,
             slab=0.366, T=0.7, thermostat="langevin", shifted=True, cutoff=2.5, dt=0.005, steps=40,
             every=20, bins=300),
        # Thermal conductivity by Fourier's law: the heat exchange on, a
        # profile and a measurement per block of steps.
        dict(name="exchange_2462", kind="exchange", n=2462, rho=0.8442, aspect=4.0, T=1.0,
             thermostat="none", shifted=True, cutoff=2.5, dt=0.002, steps=50, every=50, bins=12),
        # The production liquid: Langevin, force-shifted, 256,000 atoms.
        dict(name="liquid_256000", kind="box", n=256000, rho=0.8442, aspect=1.0, T=1.0,
             thermostat="langevin", shifted=True, cutoff=2.5, dt=0.005, steps=20),
        # The dilute million-particle fluid at constant energy.
        dict(name="fluid_1048576", kind="box", n=1048576, rho=0.4, aspect=1.0, T=1.0, thermostat="none",
             shifted=True, cutoff=2.5, dt=0.004, steps=10),
        # A few state points stepped together, every replica read at the end
        # of a block.
        dict(name="batch_32", kind="batch", count=32, lo=500, hi=20000, steps=100, read=32),
        # The equation-of-state sweep: 512 uneven replicas, measurements of
        # all of them per block, some particles looked at.
        dict(name="batch_512", kind="batch", count=512, lo=500, hi=20000, steps=20, read=2),
        # Green-Kubo: the heat current on every step of a large constant-
        # energy box (the largest case).
        dict(name="heat_current_2048000", kind="heat_current", n=2048000, rho=0.8442, aspect=1.0, T=1.0,
             thermostat="none", shifted=False, cutoff=2.5, dt=0.004, steps=20),
        # A restart from a snapshot: particles in, a short run, particles out
        # (replica exchange, parameter sweeps over one configuration).
        dict(name="restart_64000", kind="restart", n=64000, rho=0.8442, aspect=1.0, T=1.0,
             thermostat="langevin", shifted=False, cutoff=2.5, dt=0.005, steps=10),
        # Contacts of a packed bed of grains through the same cell grid.
        dict(name="grains_100000", kind="grains", n=100000, fill=0.55, spread=0.2, capacity=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box"] * 5 + ["profile", "exchange", "batch", "heat_current", "restart", "grains"])
    if kind == "grains":
        return dict(kind=kind, n=_log(rng, 2000, 200000), fill=rng.uniform(0.2, 0.6),
                    spread=rng.uniform(0.0, 0.4), capacity=rng.choice([8, 16, 24]))
    if kind == "batch":
        count = _log(rng, 3, 256)
        return dict(kind=kind, count=count, lo=rng.randint(400, 900), hi=rng.randint(3000, 20000),
                    steps=_log(rng, 5, 40), read=min(count, rng.randint(1, 6)))
    n = _log(rng, 1000, 600000 if kind in ("box", "heat_current") else 60000)
    c = dict(kind=kind, n=n, rho=rng.uniform(0.05, 0.9), aspect=1.0, T=rng.uniform(0.7, 2.0),
             thermostat="none", shifted=rng.random() < 0.5, cutoff=rng.choice([2.5, 2.5, 3.0]),
             dt=rng.choice([0.002, 0.004, 0.005]), steps=_log(rng, 4, max(5, min(60, 8000000 // n))))
    if kind in ("box", "restart", "profile"):
        c["thermostat"] = rng.choice(["none", "langevin", "nose_hoover"])
    if kind == "exchange":
        c.update(rho=rng.uniform(0.6, 0.88), n=_log(rng, 2400, 20000), aspect=4.0, shifted=True,
                 dt=0.002, cutoff=2.5)
    if kind in ("profile", "exchange"):
        c.update(bins=rng.randint(8, 300), every=max(2, c["steps"] // 2))
        c["steps"] = 2 * c["every"]
    if kind == "profile":
        c.update(n=_log(rng, 4000, 40000), aspect=rng.uniform(1.0, 4.0))
    # every side at least three (cutoff + skin) wide
    side = 3.0 * (c["cutoff"] + SKIN) * 1.01
    while _sides(c)[0] < side or _sides(c)[2] < side:
        c["n"] += c["n"] // 4 + 1
    return c


# ---- inputs, from the seed alone ----

def _sides(c):
    """Box sides (x, y, z = aspect x), rounded to f32 as the library does."""
    x = (c["n"] / c["rho"] / c["aspect"]) ** (1.0 / 3.0)
    return np.array([x, x, x * c["aspect"]]).astype(np.float32).astype(np.float64)


def _particles(n, box, T, rng, slab=None):
    """n particles on face-centred cubic sites of the box (or of its middle
    `slab` share along z), each moved a little, with Maxwell velocities at T
    and no total momentum."""
    size = np.array(box, np.float64)
    if slab:
        size[2] *= slab
    a = (4.0 * size.prod() / n) ** (1.0 / 3.0)
    m = np.maximum(1, np.rint(size / a).astype(np.int64))
    while 4 * m.prod() < n:
        m[np.argmax(size / m)] += 1
    total = int(4 * m.prod())
    site = np.arange(total) if total == n else np.sort(rng.choice(total, n, replace=False))
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    cell, b = site // 4, site % 4
    ijk = np.stack([cell % m[0], cell // m[0] % m[1], cell // (m[0] * m[1])], axis=1)
    pos = (ijk + basis[b] + 0.25) * (size / m) + rng.uniform(-0.03, 0.03, (n, 3))
    if slab:
        pos[:, 2] += 0.5 * (box[2] - size[2])
    pos = np.mod(pos, box)
    vel = rng.standard_normal((n, 3))
    vel -= vel.mean(axis=0)
    vel *= math.sqrt(T * (3 * n - 3) / (vel ** 2).sum())
    return pos, vel


def _inputs(c, seed):
    """Boxes of the case: a list of (pos, vel, sides, thermostat)."""
    rng = np.random.default_rng([int(seed), 2024])
    if c["kind"] == "batch":
        # the set of state points is the case's, the configurations the seed's
        points = np.random.default_rng([c["count"], c["lo"], c["hi"]])
        out = []
        for r in range(c["count"]):
            n = int(round(math.exp(points.uniform(math.log(c["lo"]), math.log(c["hi"])))))
            rho, T = points.uniform(0.01, 0.90), points.uniform(0.7, 2.0)
            box = np.full(3, (max(n, 620 * rho) / rho) ** (1.0 / 3.0)).astype(np.float32).astype(np.float64)
            pos, vel = _particles(n, box, T, rng)
            out.append((pos, vel, box, ("langevin", T, 1.0, (int(seed) + r) & 0xFFFFFFFF)))
        return out
    box = _sides(c)
    pos, vel = _particles(c["n"], box, c["T"], rng, c.get("slab"))
    kind = c["thermostat"]
    thermo = {"none": None, "langevin": ("langevin", c["T"], 1.0, int(seed) & 0xFFFFFFFF),
              "nose_hoover": ("nose_hoover", c["T"], 0.5)}[kind]
    return [(pos, vel, box, thermo)]


def _grains(c, seed):
    """Grains dropped on a loose lattice of a box and shaken until many touch."""
    rng = np.random.default_rng([int(seed), 77])
    r0 = 0.0015
    n = c["n"]
    radius = r0 * (1.0 + c["spread"] * rng.uniform(-1.0, 1.0, n))
    side = (n * 4.0 / 3.0 * math.pi * r0 ** 3 / c["fill"]) ** (1.0 / 3.0)
    m = math.ceil(n ** (1.0 / 3.0))
    site = np.arange(n)
    ijk = np.stack([site % m, site // m % m, site // (m * m)], axis=1)
    pos = (ijk + 0.5 + rng.uniform(-0.25, 0.25, (n, 3))) * (side / m)
    return pos, radius, side


def _thermostat(t):
    if t is None:
        return None
    return vl.Langevin(t[1], t[2], t[3]) if t[0] == "langevin" else vl.NoseHoover(t[1], t[2])


def _pinned(n):
    raw = torch.zeros(n * vl.PARTICLE.itemsize, dtype=torch.uint8, pin_memory=True)
    return raw, raw.numpy().view(vl.PARTICLE)


def _slabs(c):
    """The heat exchange's slabs: a twelfth of the box at its start and middle."""
    w = float(_sides(c)[2]) / 12.0
    return (0.0, w), (6.0 * w, 7.0 * w), 0.01


def prepare(case, seed):
    c = dict(case)
    if c["kind"] == "grains":
        pos, radius, side = _grains(c, seed)
        return dict(c=c, pos=torch.from_numpy(pos).cuda(), radius=torch.from_numpy(radius).cuda(), side=side,
                    cells=vl.grain_cells(side, float(radius.max())))
    boxes = _inputs(c, seed)
    if c["kind"] == "batch":
        reps = [vl.Replica(vl.particles(p, v), list(b), _thermostat(t)) for p, v, b, t in boxes]
        return dict(c=c, batch=vl.Batch(reps, cutoff=2.5, skin=SKIN, dt=0.004))
    pos, vel, box, t = boxes[0]
    p = vl.particles(pos, vel)
    sim = vl.LennardJones(p, vl.Settings(list(box), cutoff=c["cutoff"], dt=c["dt"], skin=SKIN,
                                         thermostat=_thermostat(t), shifted_force=c["shifted"],
                                         profile_bins=c.get("bins", 0)))
    raw, out = _pinned(c["n"])
    state = dict(c=c, sim=sim, raw=raw, out=out)
    if c["kind"] == "restart":
        state["raw_in"], state["start"] = _pinned(c["n"])
        state["start"][:] = p
    if c["kind"] == "exchange":
        hot, cold, energy = _slabs(c)
        sim.set_heat_exchange(vl.HeatExchange(hot, cold, energy))
    return state


# ---- one pass ----

def _sums(m):
    return np.array([m.kinetic, m.potential, m.virial])


def _state(state):
    out = state["sim"].read_particles(state["out"])
    return {"pos": out["pos"], "vel": out["vel"]}


def _profile(p):
    return {"slabs": np.array([[s.particles, *s.kinetic, *s.virial, s.potential] for s in p.slabs]),
            "virial": np.array(p.virial)}


def run(state):
    c = state["c"]
    kind = c["kind"]
    if kind == "grains":
        partners, counts, order, start, cell = vl.grain_contacts(
            state["pos"], state["radius"], state["side"], capacity=c["capacity"], cells=state["cells"])
        return {"partners": partners, "counts": counts, "sorted": order, "start": start, "cell": cell}
    if kind == "batch":
        b = state["batch"]
        b.run(c["steps"])
        sums = np.array([_sums(m) for m in b.measure()])
        read = [b.read_particles(r) for r in range(c["read"])]
        return {"sums": sums, "pos": np.concatenate([p["pos"] for p in read]),
                "vel": np.concatenate([p["vel"] for p in read])}
    sim = state["sim"]
    if kind in ("profile", "exchange"):
        sim.clear_profile()
        for _ in range(c["steps"] // c["every"]):
            sim.step(c["every"])
            sim.sample_profile()
        got = _profile(sim.read_profile())
        return {**got, "sums": _sums(sim.measure_now()), **_state(state)}
    if kind == "heat_current":
        sim.record_heat_current(c["steps"])
        for _ in range(c["steps"]):
            sim.sample_heat_current()
            sim.step(1)
        return {"series": sim.read_heat_current(), **_state(state)}
    if kind == "restart":
        sim.write_particles(state["start"])
    sim.run(c["steps"])
    return {"sums": _sums(sim.measure_now()), **_state(state)}


# ---- the work a pass cannot do without ----

def _flops(rho, cutoff, shifted):
    """Per particle-step: 11 for each listed neighbour, 26 (truncated 20) for
    each inside the cutoff, an FMA as two."""
    ball = 4.0 / 3.0 * math.pi * rho
    return 11.0 * ball * (cutoff + SKIN) ** 3 + (26.0 if shifted else 20.0) * ball * cutoff ** 3


def work(case):
    """Positions and velocities in f64 read and written once a step (96 B a
    particle), the arithmetic of every neighbour, and the read-back."""
    c = case
    if c["kind"] == "grains":
        cells = vl.grain_cells(*_grain_size(c)) ** 3
        # positions and radii in, the partner table, counts and grid out
        n = c["n"]
        return dict(bytes=n * (32 + 4 * c["capacity"] + 12) + 4.0 * cells, flops=n * 27 * 10.0)
    if c["kind"] == "batch":
        # N is log-uniform, the density uniform in 0.01 .. 0.90
        n = c["count"] * (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"])
        per, steps = _flops(0.455, 2.5, False), c["steps"]
        return dict(bytes=n * 96.0 * steps + n * 48.0 * c["read"] / c["count"], flops=n * per * steps)
    n, steps = c["n"], c["steps"]
    rho = c["rho"] / c.get("slab", 1.0)
    b = n * 96.0 * steps + n * 48.0
    if c["kind"] == "restart":
        b += n * 48.0
    if c["kind"] in ("profile", "exchange"):
        b += (n * 48.0 + c["bins"] * 64.0) * (steps // c["every"])
    return dict(bytes=b, flops=n * _flops(rho, c["cutoff"], c["shifted"]) * steps)


def _grain_size(c):
    r0 = 0.0015
    return ((c["n"] * 4.0 / 3.0 * math.pi * r0 ** 3 / c["fill"]) ** (1.0 / 3.0), r0 * (1.0 + c["spread"]))


def tolerance(case):
    """Forces are sums of about 50 f32 terms; the f64 state carries their
    rounding, and a few dozen steps let it grow. Against exact() velocities are
    up to 9e-7 off, sums over particles 3e-7; the heat current, a small
    difference of large terms, 1e-5. A single particle in a hard collision is
    off by more than the mean."""
    if case["kind"] == "grains":
        return "exact"
    return {"rel": 5e-5 if case["kind"] == "heat_current" else 1e-5, "max": 2e-3}


# ---- the same in 64 bits, from plain torch and numpy ----

MASK = np.uint64(0xFFFFFFFF)


def _philox(ids, step, seed):
    """Philox-4x32-10 (Salmon et al., SC'11): counter (id, step lo, step hi, 0), key (seed, "LJV1")."""
    u = np.uint64
    c = [ids.astype(u), np.full(ids.shape, step & 0xFFFFFFFF, u), np.full(ids.shape, step >> 32, u),
         np.zeros(ids.shape, u)]
    k0, k1 = seed.astype(u), np.full(ids.shape, 0x4C4A5631, u)
    for _ in range(10):
        p0, p1 = u(0xD2511F53) * c[0], u(0xCD9E8D57) * c[2]
        c = [(p1 >> u(32)) ^ c[1] ^ k0, p1 & MASK, (p0 >> u(32)) ^ c[3] ^ k1, p0 & MASK]
        k0, k1 = (k0 + u(0x9E3779B9)) & MASK, (k1 + u(0xBB67AE85)) & MASK
    return c


def _noise(ids, step, seed):
    u = [((w >> np.uint64(8)).astype(np.float64) + 1.0) / 2.0 ** 24 for w in _philox(ids, step, seed)]
    ra, rb = np.sqrt(-2.0 * np.log(u[0])), np.sqrt(-2.0 * np.log(u[2]))
    aa, ab = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return np.stack([ra * np.cos(aa), ra * np.sin(aa), rb * np.cos(ab)], axis=1)


def _half_pairs(x, box, radius):
    """Pairs i < j of one box within `radius`, through a padded cell table."""
    dev = x.device
    n = len(x)
    cells = torch.clamp((box / radius).floor().long(), min=1)
    if n < 400 or int(cells.min()) < 3:
        i, j = torch.triu_indices(n, n, 1, device=dev)
        keep = ((lambda d: d - box * torch.round(d / box))(x[j] - x[i]) ** 2).sum(1) < radius * radius
        return i[keep], j[keep]
    c = torch.minimum((x / box * cells).floor().long(), cells - 1)
    flat = (c[:, 2] * cells[1] + c[:, 1]) * cells[0] + c[:, 0]
    order = torch.argsort(flat)
    total = int(cells.prod())
    count = torch.bincount(flat, minlength=total)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    table = torch.full((total, most), -1, dtype=torch.long, device=dev)
    table[flat[order], torch.arange(n, device=dev) - start[flat[order]]] = order
    me = torch.arange(n, device=dev)
    ii, jj = [], []
    for o in range(27):
        off = torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=dev)
        t = torch.remainder(c + off, cells)
        other = table[(t[:, 2] * cells[1] + t[:, 1]) * cells[0] + t[:, 0]]
        for k in range(most):
            j = other[:, k]
            live = j > me
            i, j = me[live], j[live]
            d = x[j] - x[i]
            d = d - box * torch.round(d / box)
            keep = (d * d).sum(1) < radius * radius
            ii.append(i[keep])
            jj.append(j[keep])
    return torch.cat(ii), torch.cat(jj)


class _System:
    """Boxes side by side in f64: positions, velocities, pair forces."""

    def __init__(self, boxes, cutoff, shifted):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        put = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=self.dev)  # noqa: E731
        self.counts = [len(b[0]) for b in boxes]
        self.x = put(np.concatenate([b[0] for b in boxes]))
        self.v = put(np.concatenate([b[1] for b in boxes]))
        self.sides = [put(b[2]) for b in boxes]
        self.box = put(np.concatenate([np.broadcast_to(b[2], b[0].shape) for b in boxes]))
        self.first = np.concatenate([[0], np.cumsum(self.counts)]).astype(int)
        self.of = put(np.repeat(np.arange(len(boxes)), self.counts))
        self.rc, self.shifted, self.extra = cutoff, shifted, 0.7
        inv6 = cutoff ** -6
        self.shift = 4.0 * (inv6 * inv6 - inv6)
        self.fshift = 24.0 * (2.0 * inv6 * inv6 - inv6) / cutoff if shifted else 0.0
        self.built = None

    def lists(self):
        if self.built is not None:
            d = self.x - self.built
            d = d - self.box * torch.round(d / self.box)
            if float((d * d).sum(1).max()) < (0.49 * self.extra) ** 2:
                return
        self.built = self.x.clone()
        ii, jj = [], []
        for b in range(len(self.counts)):
            f, e = self.first[b], self.first[b + 1]
            i, j = _half_pairs(torch.remainder(self.x[f:e], self.sides[b]), self.sides[b], self.rc + self.extra)
            ii.append(i + int(f))
            jj.append(j + int(f))
        self.i, self.j = torch.cat(ii), torch.cat(jj)

    def pairs(self):
        """(i, j, d = x_j - x_i, F / r, U) of the pairs inside the cutoff."""
        self.lists()
        d = self.x[self.j] - self.x[self.i]
        side = self.box[self.i]
        d -= side * torch.round(d / side)
        r2 = (d * d).sum(1)
        keep = r2 < self.rc * self.rc
        i, j, d, r2 = self.i[keep], self.j[keep], d[keep], r2[keep]
        s6 = r2 ** -3
        r = r2.sqrt()
        f = (24.0 * (2.0 * s6 * s6 - s6) - self.fshift * r) / r2
        u = 4.0 * (s6 * s6 - s6) - self.shift + (r - self.rc) * self.fshift
        return i, j, d, f, u

    def forces(self):
        i, j, d, f, _ = self.pairs()
        a = torch.zeros_like(self.x)
        fd = d * f[:, None]
        a.index_add_(0, j, fd)
        a.index_add_(0, i, -fd)
        return a

    def sums(self):
        """Kinetic energy, potential and virial of each box."""
        i, _, d, f, u = self.pairs()
        out = torch.zeros(len(self.counts), 3, dtype=torch.float64, device=self.dev)
        out[:, 0].index_add_(0, self.of, 0.5 * (self.v ** 2).sum(1))
        out[:, 1].index_add_(0, self.of[i], u)
        out[:, 2].index_add_(0, self.of[i], f * (d * d).sum(1))
        return out.cpu().numpy()

    def heat_current(self):
        i, j, d, f, u = self.pairs()
        w = self.v[i] + self.v[j]
        return ((0.5 * (self.v ** 2).sum(1, keepdim=True) * self.v).sum(0) + (0.5 * u[:, None] * w).sum(0)
                + (0.5 * (f * (d * w).sum(1))[:, None] * d).sum(0)).cpu().numpy()

    def profile(self, bins):
        """One Irving-Kirkwood sample along z of the (single) box."""
        i, j, d, f, u = self.pairs()
        width = float(np.float32(float(self.sides[0][2]) / bins))
        # a particle's slab is that of its height rounded to f32
        z = torch.remainder(self.x[:, 2], self.box[:, 2]).float().double()
        home = torch.clamp((z / width).floor().long(), 0, bins - 1)
        out = torch.zeros(bins, 8, dtype=torch.float64, device=self.dev)
        out[:, 0].index_add_(0, home, torch.ones_like(z))
        out[:, 1:4].index_add_(0, home, self.v ** 2)
        out[:, 7].index_add_(0, home[i], 0.5 * u)
        out[:, 7].index_add_(0, home[j], 0.5 * u)
        w = d * d * f[:, None]
        lo = z[i] + torch.clamp(d[:, 2], max=0.0)
        hi = z[i] + torch.clamp(d[:, 2], min=0.0)
        length = hi - lo
        flat = length < 1e-6 * width
        share_of = torch.where(flat, torch.ones_like(length), length)
        b0 = (lo / width).floor()
        for k in range(int(math.ceil(self.rc / width)) + 2):
            b = b0 + k
            over = torch.clamp(torch.minimum(hi, (b + 1) * width) - torch.maximum(lo, b * width), min=0.0)
            share = torch.where(flat, torch.full_like(over, 1.0 if k == 0 else 0.0), over / share_of)
            out[:, 4:7].index_add_(0, torch.remainder(b, bins).long(), w * share[:, None])
        return out, w.sum(0)


def _exchange(s, a, dt, hot, cold, energy):
    """eHEX/a (Wirnsberger, Frenkel and Dellago 2015, eq. 20): heat from the cold slab to the hot one."""
    z = torch.remainder(s.x[:, 2], s.box[:, 2]).float()
    moved, scaled = torch.zeros_like(s.x), s.v.clone()
    for (lo, hi), sign in ((hot, 1.0), (cold, -1.0)):
        m = (z >= np.float32(lo)) & (z < np.float32(hi))
        k = int(m.sum())
        if not k:
            continue
        v, f = s.v[m], a[m]
        com, mean = v.mean(0), f.mean(0)
        rel = v - com
        kinetic = 0.5 * float((rel ** 2).sum())
        e = sign * float(np.float32(energy))
        flux = e / dt
        power = float((f * rel).sum())
        cv = dt ** 3 * flux / (2.0 * kinetic * kinetic) * (flux / 48.0 + power / 6.0)
        cf = dt ** 3 * flux / (12.0 * kinetic)
        moved[m] = cv * rel - cf * (f - mean)
        scaled[m] = v + (math.sqrt(1.0 + e / kinetic) - 1.0) * rel
    s.x = s.x - moved
    s.v = scaled


def exact(case, seed):
    c = case
    if c["kind"] == "grains":
        return None
    boxes = _inputs(c, seed)
    batch = c["kind"] == "batch"
    s = _System(boxes, 2.5 if batch else c["cutoff"], False if batch else c["shifted"])
    dt = 0.004 if batch else c["dt"]
    thermo = boxes[0][3]
    kind = thermo[0] if thermo else "none"
    n = len(s.x)
    if kind == "langevin":
        ids = np.concatenate([np.arange(k) for k in s.counts])
        seeds = np.concatenate([np.full(k, b[3][3]) for k, b in zip(s.counts, boxes)])
        c1 = math.exp(-thermo[2] * dt)
        T = np.concatenate([np.full((k, 1), b[3][1]) for k, b in zip(s.counts, boxes)])
        c2 = torch.as_tensor(np.sqrt((1.0 - c1 * c1) * T), device=s.dev)
    xi = 0.0
    if kind == "nose_hoover":
        gkt = (3.0 * n - 3.0) * thermo[1]
        q = gkt * thermo[2] ** 2 / (4.0 * math.pi ** 2)

    def half_thermostat():
        nonlocal xi
        ke = 0.5 * float((s.v ** 2).sum())
        xi += (2.0 * ke - gkt) / q * 0.25 * dt
        scale = math.exp(-xi * 0.5 * dt)
        s.v = s.v * scale
        xi += (2.0 * ke * scale * scale - gkt) / q * 0.25 * dt

    series, slabs, whole, samples = [], 0.0, 0.0, 0
    a = s.forces()
    for step in range(c["steps"]):
        if c["kind"] == "heat_current":
            series.append(s.heat_current())
        if kind == "nose_hoover":
            half_thermostat()
        s.v = s.v + 0.5 * dt * a
        if kind == "langevin":
            s.x = s.x + 0.5 * dt * s.v
            s.v = c1 * s.v + c2 * torch.as_tensor(_noise(ids, step, seeds), device=s.dev)
            s.x = s.x + 0.5 * dt * s.v
        else:
            s.x = s.x + dt * s.v
        a = s.forces()
        s.v = s.v + 0.5 * dt * a
        if kind == "nose_hoover":
            half_thermostat()
        if c["kind"] == "exchange":
            # the next half kick still takes the forces before the correction
            _exchange(s, a, dt, *_slabs(c))
        if c["kind"] in ("profile", "exchange") and (step + 1) % c["every"] == 0:
            one, w = s.profile(c["bins"])
            slabs, whole, samples = slabs + one, whole + w, samples + 1
    k = s.first[c["read"]] if batch else n
    out = {"pos": torch.remainder(s.x, s.box)[:k].cpu().numpy(), "vel": s.v[:k].cpu().numpy()}
    if c["kind"] == "heat_current":
        return {"series": np.array(series), **out}
    sums = s.sums()
    out["sums"] = sums if batch else sums[0]
    if c["kind"] in ("profile", "exchange"):
        out["slabs"], out["virial"] = (slabs / samples).cpu().numpy(), (whole / samples).cpu().numpy()
    return out
