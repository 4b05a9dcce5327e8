"""The work that a user of this framework has it do, as measurable cases.

Every case is a run through the public entry points (the C ABI's module
procedures and whole schedules, by way of `rmpcdmd_b200`), followed by the
copy of the particle arrays to page-locked host memory that a program makes
when it stores a snapshot:

  bulk        a bulk SRD fluid: `bulk_run`, the fused schedule
  steps       the same loop written by the user, one module procedure at a
              time (SRD or MPC-AT, reactions, observables every few intervals)
  channel     flow between two walls: gravity, wall collisions and wall
              particles, one module procedure at a time
  dimer       `single_dimer_pbc` through the replica engine (one or many)
  program     `single_dimer_pbc` as the `run` command issues it, every MD
              step a sequence of module procedures
  colloids    `n_colloids_pbc` through its native loop

Sizes are the configurations' (32^3, 96^3, 128^3 cells at density 10, 200
colloids, replica boxes of 16..48) and ragged ones of the same range.
"""
import ctypes as C
import math

import numpy as np
import torch

import rmpcdmd_b200 as rm
from rmpcdmd_b200 import programs
from rmpcdmd_b200._capi import call

RHO = 10
T0 = 1.0 / 3.0
TAU = 1.0
N_MD = 100
CHANNEL_G = 0.002
CHANNEL_BC = (1, 1, 2)  # periodic in x and y, bounce-back at the z walls


def listed():
    return [
        # a test-sized fluid, run in short blocks: launches and the latency of a call count
        dict(name="bulk_16_f64", kind="bulk", Lx=16, Ly=16, Lz=16, precision=64, intervals=10, alpha=0.0),
        # an odd box of moderate size with a rotation angle of its own
        dict(name="bulk_50_41_30_f32", kind="bulk", Lx=50, Ly=41, Lz=30, precision=32, intervals=50, alpha=2.0),
        # the bulk benchmark: 128^3 cells, 200 collision steps, both precisions
        dict(name="bulk_128_f32", kind="bulk", Lx=128, Ly=128, Lz=128, precision=32, intervals=200, alpha=0.0),
        dict(name="bulk_128_f64", kind="bulk", Lx=128, Ly=128, Lz=128, precision=64, intervals=100, alpha=0.0),
        # the user's own SRD loop with observables, in the reference's precision
        dict(name="steps_64_f64", kind="steps", Lx=64, Ly=64, Lz=64, precision=64, intervals=50, thermostat=False,
             reaction=False, sample=5),
        # a thermostatted fluid with a reversible bulk reaction
        dict(name="steps_at_90_70_50_f32", kind="steps", Lx=90, Ly=70, Lz=50, precision=32, intervals=40,
             thermostat=True, reaction=True, sample=10),
        # a thermostatted Poiseuille flow between bounce-back walls
        dict(name="channel_80_48_32_f64", kind="channel", Lx=80, Ly=48, Lz=32, precision=64, intervals=40,
             thermostat=True),
        # one dimer in a small box as the `run` command drives it, sampling the dimer twice per interval
        dict(name="program_32_f64", kind="program", Lx=32, Ly=32, Lz=32, precision=64, intervals=1, sample=50),
        # the same system in the replica engine, 1,000 MD steps
        dict(name="dimer_32_f64", kind="dimer", replicas=1, smallest=32, largest=32, precision=64, intervals=10),
        # the large-box dimer in the mixed-precision form
        dict(name="dimer_96_f32", kind="dimer", replicas=1, smallest=96, largest=96, precision=32, intervals=4),
        # an ensemble of replicas in uneven boxes
        dict(name="dimer_x48_f32", kind="dimer", replicas=48, smallest=16, largest=48, precision=32, intervals=4),
        # 200 passive colloids in 128^3 cells, thermalisation loops
        dict(name="colloids_128_f32", kind="colloids", Lx=128, Ly=128, Lz=128, precision=32, intervals=10,
             colloids=200, thermostat=True),
    ]


def _box(rng, lo, hi):
    """Three sides of a box whose number of cells is log-uniform between lo and hi."""
    side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1 / 3)
    f, g = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    return [max(4, round(side * f)), max(4, round(side * g)), max(4, round(side / (f * g)))]


def draw(rng):
    kind = rng.choice(["bulk", "steps", "channel", "dimer", "program", "colloids"])
    precision = rng.choice([32, 64])
    if kind in ("bulk", "steps", "channel"):
        L = _box(rng, 16 ** 3, 120 ** 3 if kind == "bulk" else 80 ** 3)
        case = dict(kind=kind, Lx=L[0], Ly=L[1], Lz=L[2], precision=precision, intervals=rng.randint(10, 60))
        if kind == "bulk":
            case["alpha"] = rng.choice([0.0, 1.0, 2.0, 2.27])
        else:
            case["thermostat"] = rng.choice([True, False])
        if kind == "steps":
            case["reaction"] = rng.choice([True, False])
            case["sample"] = rng.choice([1, 5, 10])
        return case
    if kind == "dimer":
        lo = rng.choice([16, 20, 24, 32, 40, 48, 72])
        hi = min(80, lo + rng.choice([0, 8, 16]))
        most = max(1, 20000000 // (RHO * hi ** 3))
        n = min(most, round(math.exp(rng.uniform(0, math.log(64)))))
        return dict(kind=kind, replicas=n, smallest=lo, largest=hi, precision=precision, intervals=rng.randint(1, 4))
    if kind == "program":
        L = _box(rng, 18 ** 3, 64 ** 3)
        return dict(kind=kind, Lx=max(16, L[0]), Ly=max(16, L[1]), Lz=max(16, L[2]), precision=precision, intervals=1,
                    sample=rng.choice([10, 25, 50]))
    L = _box(rng, 48 ** 3, 110 ** 3)
    L = [max(38, x) for x in L]
    n = max(1, round(L[0] * L[1] * L[2] * math.exp(rng.uniform(math.log(2e-5), math.log(2e-4)))))
    return dict(kind=kind, Lx=L[0], Ly=L[1], Lz=L[2], precision=precision, intervals=rng.randint(1, 5), colloids=n,
                thermostat=rng.choice([True, False]))


# ------------------------------------------------------------------ inputs
def _inputs(case, seed):
    """Uniform positions and Maxwell velocities of zero total momentum, made from the seed on the GPU."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    n = RHO * case["Lx"] * case["Ly"] * case["Lz"]
    edges = torch.tensor([case["Lx"], case["Ly"], case["Lz"]], dtype=torch.float64, device=dev)
    pos = torch.rand(n, 3, generator=g, dtype=torch.float64, device=dev) * edges
    vel = torch.randn(n, 3, generator=g, dtype=torch.float64, device=dev) * math.sqrt(T0)
    vel -= vel.mean(0)
    return n, pos, vel


def _snapshot_buffers(n, int_fields):
    """Page-locked arrays for the fields of a snapshot."""
    out = {f: torch.empty(n, 3, dtype=torch.float64, pin_memory=True).numpy() for f in ("pos", "vel")}
    for f in int_fields:
        shape = (n, 3) if f == "image" else (n,)
        out[f] = torch.empty(*shape, dtype=torch.int32, pin_memory=True).numpy()
    return out


def _snapshot(p, buffers, first=0):
    """The particle arrays of p into rows first.. of the page-locked arrays."""
    for f, a in buffers.items():
        call("rmpcd_particles_download", p.handle, f.encode(), C.c_void_p(a.ctypes.data + first * a.strides[0]))


def _fluid(case, seed):
    L = [case["Lx"], case["Ly"], case["Lz"]]
    walls = case["kind"] == "channel"
    n, pos, vel = _inputs(case, seed)
    s = {"cells": rm.CellSystem(L, 1.0, has_walls=walls), "rng": rm.Rng(seed)}
    reacting = case.get("reaction", False)
    s["p"] = p = rm.ParticleSystem(n, 2 if reacting else 1, None, case["precision"])
    p.pos = pos.cpu().numpy()
    p.vel = vel.cpu().numpy()
    p.species = np.arange(n, dtype=np.int32) % 2 + 1 if reacting else 1
    if reacting:
        s["cells"].is_reac = np.ones(s["cells"].N, np.uint8)
    if walls:
        s["cells"].set_bc(CHANNEL_BC)
    s["cells"].random_shift(s["rng"])
    p.sort(s["cells"])
    s["snapshot"] = _snapshot_buffers(n, ("species", "id") if reacting else ("image", "id"))
    return s


def _sides(case):
    """The box sides of the replicas: the usual ones of the range in turn, the largest first."""
    sizes = [x for x in (96, 80, 72, 64, 56, 48, 40, 32, 24, 20, 16) if case["smallest"] <= x <= case["largest"]]
    return [sizes[k % len(sizes)] for k in range(case["replicas"])]


def _dimers(case, seed):
    d = [programs.SingleDimerPBC(L=(x, x, x), rho=RHO, T=T0, tau=TAU, N_MD=N_MD, seed=seed * 1000 + k,
                                 list_capacity=4000, precision=case["precision"]) for k, x in enumerate(_sides(case))]
    s = {"batch": programs.DimerBatch(d), "dimers": d}
    s["snapshot"] = _snapshot_buffers(sum(x.N for x in d), ("species",))
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("bulk", "steps", "channel"):
        s = _fluid(case, seed)
    elif kind == "dimer":
        s = _dimers(case, seed)
    elif kind == "program":
        L = (case["Lx"], case["Ly"], case["Lz"])
        d = programs.SingleDimerPBC(L=L, rho=RHO, T=T0, tau=TAU, N_MD=N_MD, seed=seed, list_capacity=4000,
                                    precision=case["precision"])
        s = {"dimer": d, "snapshot": _snapshot_buffers(d.N, ("species",))}
    else:
        L = (case["Lx"], case["Ly"], case["Lz"])
        g = programs.NColloidsPBC(L=L, rho=RHO, T=T0, tau=TAU, N_MD=N_MD, N_colloids=case["colloids"], seed=seed,
                                  precision=case["precision"], volume_correction=False)
        s = {"colloids": g, "snapshot": _snapshot_buffers(g.N, ("id",))}
    s["case"] = case
    return s


# -------------------------------------------------------------------- runs
def _run_bulk(s, case):
    rm.bulk_run(s["p"], s["cells"], s["rng"], TAU, case["intervals"], alpha=case["alpha"] or None)
    _snapshot(s["p"], s["snapshot"])
    return dict(s["snapshot"])


def _run_steps(s, case):
    p, c, rng = s["p"], s["cells"], s["rng"]
    temperature, sums = [], []
    for k in range(1, case["intervals"] + 1):
        rm.simple_mpcd_step(p, c, rng, thermostat=case["thermostat"], T=T0)
        if case["reaction"]:
            rm.bulk_reaction(p, c, 1, 2, 0.01, TAU, rng)
            rm.bulk_reaction(p, c, 2, 1, 0.01, TAU, rng)
        rm.mpcd_stream_periodic(p, c, TAU)
        c.random_shift(rng)
        p.sort(c)
        if k % case["sample"] == 0:
            temperature.append(rm.compute_temperature(p, c))
            sums.append(rm.velocity_sums(p))
    _snapshot(p, s["snapshot"])
    return dict(s["snapshot"], temperature=np.array(temperature), sums=np.array(sums)[:, 0])


def _run_channel(s, case):
    p, c, rng = s["p"], s["cells"], s["rng"]
    for _ in range(case["intervals"]):
        rm.mpcd_stream_xforce_yzwall(p, c, TAU, CHANNEL_G)
        rm.apply_pbc(p, c.edges)
        c.random_shift(rng)
        p.sort(c)
        rm.wall_mpcd_step(p, c, rng, wall_temperature=[T0, T0], wall_v=np.zeros((3, 2)), wall_n=[RHO, RHO],
                          thermostat=case["thermostat"], bulk_temperature=T0)
    _snapshot(p, s["snapshot"])
    return dict(s["snapshot"], temperature=rm.compute_temperature(p, c))


def _run_dimer(s, case):
    b, dimers = s["batch"], s["dimers"]
    b.run(case["intervals"])
    first = 0
    cpos, cvel = [], []
    for r, d in enumerate(dimers):
        b.scatter(r)
        _snapshot(d.solvent, s["snapshot"], first)
        first += d.N
        cpos.append(d.colloids.pos)
        cvel.append(d.colloids.vel)
    return dict(s["snapshot"], colloid_pos=np.array(cpos), colloid_vel=np.array(cvel),
                extra_sorting=np.asarray(b.n_extra_sorting()))


def _run_program(s, case):
    d = s["dimer"]
    out = {"position": [], "velocity": [], "image": [], "n_solvent": [], "temperature": [], "internal": []}
    for _ in range(case["intervals"]):
        for j in range(1, N_MD + 1):
            d.md_step(want_energy=j == N_MD)
            if j % case["sample"] == 0:
                out["position"].append(d.colloids.pos)
                out["velocity"].append(d.colloids.vel)
                out["image"].append(d.colloids.image)
        th = d.thermo()
        out["temperature"].append(th["temperature"])
        out["internal"].append(th["internal"])
        d.mpcd()
        out["n_solvent"].append(rm.n_solvent(d.solvent, 2))
    _snapshot(d.solvent, s["snapshot"])
    return dict(s["snapshot"], **{k: np.array(v) for k, v in out.items()})


def _run_colloids(s, case):
    g = s["colloids"]
    if case["thermostat"]:
        g.thermalise(case["intervals"])
    else:
        g.run(case["intervals"])
    _snapshot(g.solvent, s["snapshot"])
    return dict(s["snapshot"], colloid_pos=g.colloids.pos, colloid_vel=g.colloids.vel,
                temperature=rm.compute_temperature(g.solvent, g.cells), energies=np.array([g.e1, g.e2]))


_RUN = {"bulk": _run_bulk, "steps": _run_steps, "channel": _run_channel, "dimer": _run_dimer,
        "program": _run_program, "colloids": _run_colloids}


def run(state):
    case = state["case"]
    return _RUN[case["kind"]](state, case)


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: positions and velocities read and written once in every interval and, with MD steps, positions
    read and written and velocities read in every MD step (of the solvent near the colloids only in the
    lazily streamed `colloids`), and the snapshot; operations of the collision, streaming and key of a
    particle, about 100, and of an MD step, about 20."""
    w = case["precision"] // 8
    if case["kind"] == "dimer":
        n = RHO * sum(x ** 3 for x in _sides(case))
    else:
        n = RHO * case["Lx"] * case["Ly"] * case["Lz"]
    k = case["intervals"]
    moved, ops = 12 * w * n * k + 48 * n, 100.0 * n * k
    if case["kind"] in ("dimer", "program"):
        moved += 9 * w * n * N_MD * k
        ops += 20.0 * n * N_MD * k
    elif case["kind"] == "colloids":
        near = min(n, case["colloids"] * RHO * 4 / 3 * math.pi * 5.0 ** 3)
        moved += 9 * w * near * N_MD * k
        ops += 20.0 * near * N_MD * k
    return {"bytes": moved, "flops": ops}


# ------------------------------------------------------------------- exact
# The loops of `bulk`, `steps` and `channel` once more in 64-bit torch: Philox4x32-10 (Salmon et al., SC'11)
# draws addressed by (index, step, stream, attempt), Marsaglia's unit vectors, Leva's normals, Hamilton's
# compact Hilbert order of the cells.  An FP32 run leaves it as soon as one particle's rounding puts it
# into another cell, and the dimer and colloid programs are chaotic: they have no such value.
_SHIFT, _AXIS, _GAUSS = 1, 2, 3
_M32 = 0xFFFFFFFF


def _philox(c, key):
    c0, c1, c2, c3 = c
    k0, k1 = key & _M32, (key >> 32) & _M32
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & _M32) ^ c1 ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c3 ^ k1, p0 & _M32
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


def _uniform2(seed, step, index, stream, attempt):
    last = torch.full_like(index, (stream << 24) | attempt)
    o = _philox((index, torch.full_like(index, step & _M32), torch.full_like(index, step >> 32), last), seed)
    # 53 of 64 bits: all of the high word, 21 bits of the low one
    return [(o[k + 1] * (1 << 21) + (o[k] >> 11)).double() / (1 << 53) for k in (0, 2)]


def _shift(seed, step, dev):
    i = torch.arange(2, dtype=torch.int64, device=dev)
    a, b = _uniform2(seed, step, i, _SHIFT, 0)
    return torch.stack([a[0], b[0], a[1]]) - 1


def _accepted(attempt, n, width, most, dev):
    """The first accepted of attempts 0, 1, ... for each of n draws."""
    out = torch.zeros(n, width, dtype=torch.float64, device=dev)
    left = torch.arange(n, dtype=torch.int64, device=dev)
    for t in range(most):
        ok, z = attempt(left, t)
        out[left[ok]] = z[ok]
        left = left[~ok]
        if not len(left):
            break
    return out


def _axes(seed, step, n, dev):
    def attempt(i, t):
        a, b = _uniform2(seed, step, i, _AXIS, t)
        x, y = 2 * a - 1, 2 * b - 1
        s = x * x + y * y
        f = 2 * torch.sqrt((1 - s).clamp(min=0))
        return s < 1, torch.stack([x * f, y * f, 1 - 2 * s], 1)
    return _accepted(attempt, n, 3, 64, dev)


def _normals(seed, step, n, first, dev):
    """Columns first, first + 1, first + 2 of the normal deviates of indices 0 .. n - 1."""
    def one(sub):
        def attempt(i, t):
            a, b = _uniform2(seed, step, i, _GAUSS, (sub << 16) | t)
            u, v = 1 - a, 1.7156 * (b - 0.5)
            x, y = u - 0.449871, v.abs() + 0.386595
            q = x * x + y * (0.19600 * y - 0.25472 * x)
            return (q < 0.27597) | ((q <= 0.27846) & (v * v <= -4 * torch.log(u) * u * u)), (v / u)[:, None]
        return _accepted(attempt, n, 1, 256, dev)
    return torch.cat([one(first + k) for k in range(3)], 1)


def _hilbert_order(L):
    """Compact Hilbert index of every cell, p0 + L0 (p1 + L1 p2), and the number of indices."""
    M = [max(1, math.ceil(math.log2(x))) for x in L]
    p = [x.reshape(-1) for x in np.meshgrid(*[np.arange(x) for x in L], indexing="ij")]
    h = np.zeros(len(p[0]), np.int64)
    e, d = np.zeros_like(h), np.full_like(h, 2)

    def right(x, r):
        return ((x >> r) | (x << (3 - r))) & 7

    def left(x, r):
        return ((x << r) | (x >> (3 - r))) & 7

    gray = np.array([i ^ (i >> 1) for i in range(8)])
    back = np.argsort(gray)
    entry = np.array([0] + [gray[2 * ((i - 1) // 2)] for i in range(1, 8)])
    flips = [int(math.log2((i ^ (i >> 1)) ^ ((i + 1) ^ ((i + 1) >> 1)))) for i in range(8)]
    turn = np.array([0] + [flips[i if i % 2 else i - 1] % 3 for i in range(1, 8)])
    for i in range(max(M) - 1, -1, -1):
        active = sum(1 << k for k in range(3) if M[k] > i)
        rot = (d + 1) % 3
        mask = right(np.full_like(h, active), rot)
        word = sum(((p[k] >> i) & 1) << k for k in range(3))
        w = back[right(word ^ e, rot)]
        for b in (2, 1, 0):
            h = np.where((mask >> b) & 1, (h << 1) | ((w >> b) & 1), h)
        e = e ^ left(entry[w], rot)
        d = (d + turn[w] + 1) % 3
    table = np.empty(len(h), np.int64)
    table[p[0] + L[0] * (p[1] + L[1] * p[2])] = h
    return table, 1 << sum(M)


class _Fluid64:
    """Positions, velocities and cells in 64 bits."""

    def __init__(self, case, seed):
        self.n, self.pos, self.vel = _inputs(case, seed)
        self.dev, self.seed = self.pos.device, seed & 0xFFFFFFFFFFFFFFFF
        self.walls = case["kind"] == "channel"
        self.L = [case["Lx"], case["Ly"], case["Lz"]]
        self.edges = torch.tensor(self.L, dtype=torch.float64, device=self.dev)
        cells = [self.L[0], self.L[1], self.L[2] + (1 if self.walls else 0)]
        self.grid = torch.tensor(cells, dtype=torch.int64, device=self.dev)
        table, self.S = _hilbert_order(cells)
        self.table = torch.from_numpy(table).to(self.dev)
        if self.walls:
            z = torch.arange(len(table), device=self.dev) // (cells[0] * cells[1])
            self.wall_cell = torch.zeros(self.S, dtype=torch.bool, device=self.dev)
            self.wall_cell[self.table] = (z == 0) | (z == cells[2] - 1)
        self.step = 0
        self.shift_and_sort()

    def shift_and_sort(self):
        c = torch.floor(self.pos - _shift(self.seed, self.step, self.dev)).to(torch.int64)
        self.step += 1
        around = c == self.grid
        if self.walls:
            around[:, 2] = False
        c = torch.where(around, torch.zeros_like(c), c)
        key = self.table[c[:, 0] + self.grid[0] * (c[:, 1] + self.grid[1] * c[:, 2])]
        self.slot, order = torch.sort(key, stable=True)
        self.pos, self.vel = self.pos[order], self.vel[order]
        self.count = torch.bincount(self.slot, minlength=self.S)
        self.many = (self.count > 1)[self.slot][:, None]

    def cell_sum(self, v):
        return torch.zeros(self.S, v.shape[1], dtype=torch.float64, device=self.dev).index_add_(0, self.slot, v)

    def collide(self, thermostat, alpha=0.0):
        n = self.count[:, None].clamp(min=1).double()
        mean = self.cell_sum(self.vel) / n
        if self.walls:
            short = self.wall_cell & (self.count < RHO)
            virtual = _normals(self.seed, self.step, self.S, 3, self.dev)
            virtual *= torch.sqrt((RHO - self.count).clamp(min=0).double() * T0)[:, None]
            mean = torch.where(short[:, None], (mean * n + virtual) / RHO, mean)
        if thermostat:
            new = _normals(self.seed, self.step, self.n, 0, self.dev) * math.sqrt(T0)
            new = new + (mean - self.cell_sum(new) / n)[self.slot]
        else:
            sin_a, cos_a = (math.sin(alpha), math.cos(alpha)) if alpha else (1.0, 0.0)
            a, m = _axes(self.seed, self.step, self.S, self.dev)[self.slot], mean[self.slot]
            r = self.vel - m
            # the rotation matrix of the collision turns r by -alpha about the axis
            new = m + cos_a * r + (1 - cos_a) * (a * r).sum(1, keepdim=True) * a + sin_a * torch.cross(r, a, dim=1)
        self.vel = torch.where(self.many, new, self.vel)
        self.step += 1

    def stream(self):
        self.pos = self.pos + self.vel * TAU
        self.pos = self.pos - torch.floor(self.pos / self.edges) * self.edges

    def stream_channel(self):
        """Gravity along x; a particle that meets a z wall turns back there and goes on for the time left."""
        g = torch.tensor([CHANNEL_G, 0.0, 0.0], dtype=torch.float64, device=self.dev)
        end = self.pos + self.vel * TAU + g * TAU ** 2 / 2
        vz, z, Lz = self.vel[:, 2], self.pos[:, 2], float(self.L[2])
        hit = ((end[:, 2] < 0) | (end[:, 2] > Lz))[:, None]
        t = (torch.where(vz > 0, Lz - z, -z) / vz)[:, None]
        left = TAU - t
        v = -(self.vel + g * t)
        turned = self.pos + self.vel * t + g * t * t / 2 + v * left + g * left * left / 2
        # a free particle keeps its velocity: the reference adds the field's only in wall collisions
        self.vel = torch.where(hit, v + g * left, self.vel)
        self.pos = torch.where(hit, turned, end)
        self.pos = self.pos - torch.floor(self.pos / self.edges) * self.edges

    def temperature(self):
        mean = self.cell_sum(self.vel) / self.count[:, None].clamp(min=1)
        kin = self.cell_sum(((self.vel - mean[self.slot]) ** 2).sum(1, keepdim=True))[:, 0]
        on = self.count > 1
        return float((kin[on] / (3 * (self.count[on] - 1))).mean())


def exact(case, seed):
    if case["precision"] == 32 or case["kind"] not in ("bulk", "steps", "channel"):
        return None
    f = _Fluid64(case, seed)
    out = {"pos": None, "vel": None, "image": None, "id": None}
    if case.get("reaction"):
        out = {"pos": None, "vel": None, "species": None, "id": None}
    temperature, sums = [], []
    for k in range(1, case["intervals"] + 1):
        if case["kind"] == "channel":
            f.stream_channel()
            f.shift_and_sort()
            f.collide(case["thermostat"])
            continue
        f.collide(case.get("thermostat", False), case.get("alpha", 0.0))
        if case.get("reaction"):
            f.step += 2
        f.stream()
        f.shift_and_sort()
        if case["kind"] == "steps" and k % case["sample"] == 0:
            temperature.append(f.temperature())
            sums.append(float((f.vel ** 2).sum()))
    out["pos"], out["vel"] = f.pos, f.vel
    if case["kind"] == "steps":
        out.update(temperature=np.array(temperature), sums=np.array(sums))
    elif case["kind"] == "channel":
        out["temperature"] = f.temperature()
    return out
