"""The work that users of this library have it do, as cases that can be timed.

A pass is a stretch of a running simulation: some steps through ``Selm.run``
or ``Batch.run``, then the monomers read back as a trajectory writer or an
analysis reads them.  ``prepare`` makes the system (chains grown from the
seed, Maxwell velocities), starts it and takes ``WARM`` steps, as every pass
stands for a part of a run of thousands.  Results of the FP32 form are kept in
float32, the precision of its fluid and of a DCD frame; those of the FP64
forms in float64.

``exact`` is the same run in plain torch, in 64 bits: the step written from
its equations (spectral fluid update, Peskin interpolation and spreading,
explicit monomer update, bonds, angles and pairs) with the Philox draws that
the library documents.
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from monomers2026_b200 import _lib
from monomers2026_b200.analysis import Analysis
from monomers2026_b200.selm import Batch, Params, Selm, Topology
from monomers2026_b200.workloads import fene_wca_topology, harmonic_chain_topology

WARM = 2  # steps taken by prepare: both parities of the double-buffered positions
RUN, BATCH, ROUND_TRIP = "run", "batch", "round trip"


def listed():
    return [
        # The smallest call: configuration 1, one harmonic chain of 20 in the
        # reference's own form (FP64, one kernel per reference kernel).
        dict(name="chain32_plain64", kind=RUN, form="plain64", integrator="inertial", noise="ref_compat", grid=32,
             system="harmonic", chains=1, length=20, kT=1.0, steps=20, field=True, sample=False),
        # The reference's example case: 96 four-bead nucleotides with bonds,
        # angles and pairs on 30^3, in the fused FP64 form.
        dict(name="nucleotides30_fused64", kind=RUN, form="fused64", integrator="inertial", noise="ref_compat", grid=30,
             system="nucleotides", chains=96, length=4, kT=2.479, steps=20, field=True, sample=False),
        # Configuration 2 in its two forms: 10 FENE chains of 100 on 64^3; the
        # FP32 run samples MSD and S(q) on the device as a production run does.
        dict(name="fene64_fused32", kind=RUN, form="fused32", integrator="inertial", noise="ref_compat", grid=64,
             system="fene", chains=10, length=100, kT=1.0, steps=20, field=False, sample=True),
        dict(name="fene64_plain64", kind=RUN, form="plain64", integrator="inertial", noise="ref_compat", grid=64,
             system="fene", chains=10, length=100, kT=1.0, steps=20, field=False, sample=False),
        # Configuration 3, the headline: 1000 FENE chains of 100 on 128^3 in
        # the throughput form, the accuracy form and the reference's form.
        dict(name="fene128_fused32", kind=RUN, form="fused32", integrator="inertial", noise="ref_compat", grid=128,
             system="fene", chains=1000, length=100, kT=1.0, steps=20, field=False, sample=False),
        dict(name="fene128_fused64", kind=RUN, form="fused64", integrator="inertial", noise="ref_compat", grid=128,
             system="fene", chains=1000, length=100, kT=1.0, steps=20, field=False, sample=False),
        dict(name="fene128_plain64", kind=RUN, form="plain64", integrator="inertial", noise="ref_compat", grid=128,
             system="fene", chains=1000, length=100, kT=1.0, steps=10, field=False, sample=False),
        # The overdamped form of the same system.
        dict(name="quasi128_fused32", kind=RUN, form="fused32", integrator="quasi_steady", noise="exact", grid=128,
             system="fene", chains=1000, length=100, kT=1.0, steps=20, field=False, sample=False),
        # A box whose side is no power of two and no whole number of spread
        # tiles, with the Hermitian-exact noise.
        dict(name="fene100_fused32", kind=RUN, form="fused32", integrator="inertial", noise="exact", grid=100,
             system="fene", chains=300, length=100, kT=1.0, steps=20, field=False, sample=False),
        # The largest: twice the headline's monomers in a box half again as wide.
        dict(name="fene192_fused32", kind=RUN, form="fused32", integrator="inertial", noise="ref_compat", grid=192,
             system="fene", chains=2000, length=100, kT=1.0, steps=10, field=False, sample=False),
        # An ensemble of uneven replicas stepped together (configuration 4's
        # ranges; 48 is what the serving configuration holds at a time).
        dict(name="ensemble48_fused32", kind=BATCH, form="fused32", integrator="inertial", noise="ref_compat", mix=1004,
             replicas=48, steps=10),
        # A host MD code that owns the monomers: every step uploads positions
        # and velocities from pinned memory and reads the monomers back.
        dict(name="host_round_trip128_fused64", kind=ROUND_TRIP, form="fused64", integrator="inertial",
             noise="ref_compat", grid=128, system="fene", chains=1000, length=100, kT=1.0, steps=4, field=False,
             sample=False),
    ]


def _grid_ok(n):
    for p in range(2, 62):
        while n % p == 0:
            n //= p
    return n == 1


def draw(rng):
    kind = rng.choices((RUN, BATCH, ROUND_TRIP), (8, 1, 1))[0]
    form = rng.choices(("fused32", "fused64", "plain64"), (5, 3, 2))[0]
    integrator = "inertial" if form == "plain64" or rng.random() < 0.75 else "quasi_steady"
    noise = rng.choice(("ref_compat", "exact"))
    if kind == BATCH:
        return dict(kind=BATCH, form="fused32" if form == "plain64" else form, integrator=integrator, noise=noise,
                    mix=rng.randrange(1 << 30), replicas=rng.randint(2, 24), steps=rng.randint(4, 10))
    most = {"fused32": 176, "fused64": 128, "plain64": 120}[form]
    while True:
        grid = int(round(math.exp(rng.uniform(math.log(16), math.log(most)))))
        if _grid_ok(grid):
            break
    # up to 0.04 monomers a cell (the headline has 0.048), in chains of 20 to 100
    length = rng.choice((20, 50, 100))
    top = max(2.0, 0.04 * grid ** 3 / length)
    chains = max(1, int(math.exp(rng.uniform(0.0, math.log(top)))))
    system = "harmonic" if chains * length <= 400 and rng.random() < 0.5 else "fene"
    kT = rng.choice((0.0, 0.5, 1.0, 1.0))
    return dict(kind=kind, form=form, integrator=integrator, noise=noise, grid=grid, system=system, chains=chains,
                length=length, kT=kT, steps=rng.randint(1, 6 if kind == ROUND_TRIP else 20), field=grid <= 48,
                sample=kind == RUN and rng.random() < 0.25)


# ---------------------------------------------------------------- inputs
def _grow(rng, chains, length, L, min_sep=0.95):
    """Self-avoiding random walks of unit steps in the periodic box [0, L):
    every chain grows a bead at a time, all of them at once.  A cell holds one
    bead at most (its diagonal is below min_sep)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nc = math.ceil(L * math.sqrt(3.0) / min_sep) + 1
    cell = torch.full((nc ** 3,), -1, dtype=torch.int64, device=dev)
    off = torch.arange(-2, 3, device=dev)
    off = torch.stack(torch.meshgrid(off, off, off, indexing="ij"), -1).reshape(1, -1, 3)
    x = torch.zeros((chains * length, 3), dtype=torch.float64, device=dev)
    have = torch.zeros(chains, dtype=torch.int64, device=dev)
    failed = torch.zeros_like(have)
    first = torch.arange(chains, device=dev) * length

    def at(c):
        c = torch.remainder(c, nc)
        return (c[..., 2] * nc + c[..., 1]) * nc + c[..., 0]

    def cells(p):
        return torch.clamp((p / L * nc).long(), 0, nc - 1)

    while True:
        who = torch.nonzero(have < length).reshape(-1)
        if not len(who):
            return x.cpu().numpy()
        step = rng.standard_normal((len(who), 3))
        step = torch.from_numpy(step / np.linalg.norm(step, axis=1, keepdims=True)).to(dev)
        origin = torch.from_numpy(rng.random((len(who), 3)) * L).to(dev)
        tip = x[torch.clamp(first[who] + have[who] - 1, min=0)]
        p = torch.remainder(torch.where((have[who] == 0)[:, None], origin, tip + step), L)
        near = cell[at(cells(p)[:, None, :] + off)]
        d = p[:, None, :] - x[torch.clamp(near, min=0)]
        d = d - L * torch.round(d / L)
        ok = ~((near >= 0) & ((d * d).sum(-1) < min_sep ** 2)).any(1)
        # of new beads too close to each other the first stays
        d = p[:, None, :] - p[None, :, :]
        d = d - L * torch.round(d / L)
        close = (d * d).sum(-1) < min_sep ** 2
        ok &= ~(torch.tril(close, -1) & ok[None, :]).any(1)
        new = first[who[ok]] + have[who[ok]]
        x[new] = p[ok]
        cell[at(cells(p[ok]))] = new
        have[who[ok]] += 1
        failed[who] += 1
        failed[who[ok]] = 0
        for c in torch.nonzero(failed > 40).reshape(-1).tolist():  # shut in: the chain's last beads go
            n = int(have[c])
            gone = torch.arange(max(0, n - 5), n, device=dev) + int(first[c])
            cell[at(cells(x[gone]))] = -1
            have[c] = max(0, n - 5)
            failed[c] = 0


def _nucleotides(rng, molecules):
    """Four-bead molecules (three bonds, three angles) at the sites of a
    lattice in the [-3, 3] box, with the example case's units and constants."""
    shape = np.array([[0.0, 0.0, 0.0], [0.0, -0.63, 0.0], [0.32, -0.92, 0.0], [-0.32, -0.92, 0.28]])
    site = np.stack(np.meshgrid(np.arange(5), np.arange(5), np.arange(5), indexing="ij"), -1).reshape(-1, 3)
    site = site[rng.permutation(len(site))[:molecules]] * 1.2 - 2.4
    x = site[:, None, :] + shape[None] + rng.normal(0.0, 0.004, (molecules, 4, 3)) + rng.random(3) * 0.2
    x = -3.0 + np.mod(x.reshape(-1, 3) + 3.0, 6.0)
    b, a = [], []
    for q in range(molecules):
        o = 4 * q
        b += [(1, o, o + 1), (2, o + 1, o + 2), (3, o + 1, o + 3)]
        a += [(1, o, o + 1, o + 3), (2, o, o + 1, o + 2), (3, o + 2, o + 1, o + 3)]
    sigma = np.array([0.5, 0.542, 0.422, 0.488])
    pair = np.zeros((5, 5, 3))
    for i in range(4):
        for j in range(4):
            s = 0.5 * (sigma[i] + sigma[j])
            pair[i + 1, j + 1] = (1.0, s, s)
    topo = Topology(types=np.tile(np.arange(1, 5, dtype=np.int32), molecules), ntypes=4, bonds=np.array(b, np.int32),
                    bond_style="harmonic",
                    bond_coeff=np.array([[0, 0, 0, 0], [9934.817, 0.7, 0, 0], [2250.785, 0.456, 0, 0],
                                         [4860.383, 0.502, 0, 0]], float),
                    angles=np.array(a, np.int32), angle_style="harmonic",
                    angle_coeff=np.array([[0, 0], [51.084, 99.085], [27.469, 128.857], [37.735, 106.014]], float),
                    pair_style="lj/cut", pair_coeff=pair.reshape(-1, 3))
    return x, np.tile([214.0, 83.0, 217.0, 319.0], molecules), topo


def _system(case, seed):
    """(params, x, v, mass, topology) of a case's simulation."""
    rng = np.random.default_rng(seed)
    n, kT = int(case["grid"]), float(case["kT"])
    common = dict(numMeshPtsPerDir=(n, n, n), flagStochasticDriving=int(kT > 0), SELM_Seed=int(seed), form=case["form"],
                  integrator=case["integrator"], noise_mode=case["noise"])
    if case["system"] == "nucleotides":
        x, mass, topo = _nucleotides(rng, case["chains"])
        par = Params(box_lo=-3.0, box_hi=3.0, rho=493.936086, mu=752.767749, KB=1.0, T=kT, dt=0.001, **common)
    else:
        x = _grow(rng, case["chains"], case["length"], float(n))
        mass = np.ones(len(x))
        make = harmonic_chain_topology if case["system"] == "harmonic" else fene_wca_topology
        # without thermal driving a body force moves the chains
        topo = make(case["chains"], case["length"], body=(0.0 if kT > 0 else 0.01, 0.0, 0.0))
        par = Params(box_lo=0.0, box_hi=float(n), rho=1.0, mu=1.0, KB=1.0, T=kT,
                     dt=0.01 if case["system"] == "harmonic" else 0.005, **common)
    v = rng.standard_normal(x.shape) * np.sqrt(max(kT, 0.25) / mass)[:, None]
    return par, x, v, mass, topo


def _members(case):
    """The replicas of an ensemble, from the case alone: grid, monomers and
    temperature in configuration 4's ranges, chains of 50."""
    r = random.Random(case["mix"])
    got = []
    for _ in range(case["replicas"]):
        grid = r.choice((32, 48, 64, 96))
        M = math.exp(r.uniform(math.log(50), math.log(min(2000, 0.04 * grid ** 3))))
        got.append(dict(form=case["form"], integrator=case["integrator"], noise=case["noise"], grid=grid, system="fene",
                        chains=max(1, round(M / 50)), length=50, kT=r.uniform(0.5, 2.0)))
    return got


QVEC = ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1), (2, 0, 0))
NLAG = 10


def prepare(case, seed):
    if case["kind"] == BATCH:
        sims = []
        batch = Batch()
        for k, m in enumerate(_members(case)):
            par, x, v, mass, topo = _system(m, 1000 * seed + k)
            sim = Selm(par, x, mass, v=v, topology=topo)
            sim.initial()
            batch.add(sim)
            sims.append(sim)
        batch.run(WARM)
        batch.synchronize()
        return dict(case=case, batch=batch, sims=sims)
    par, x, v, mass, topo = _system(case, seed)
    sim = Selm(par, x, mass, v=v, topology=topo)
    sim.initial()
    sim.run(WARM)
    sim.synchronize()
    state = dict(case=case, sim=sim)
    if case["kind"] == ROUND_TRIP:
        # the host code's own arrays, page-locked
        for k in "xvf":
            state[k] = torch.zeros((len(x), 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        _read(sim, state["x"], state["v"], state["f"])
    if case["sample"]:
        state["analysis"] = Analysis(sim, nlag=NLAG, lag_stride=1, qvec=np.array(QVEC))
        state["analysis"].sample()
    return state


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _read(sim, x, v, f):
    _lib.check(_lib.load().selm_get_particles(sim._h, _ptr(x), _ptr(v), _ptr(f)))


# ---------------------------------------------------------------- a pass
def run(state):
    case = state["case"]
    if case["kind"] == BATCH:
        state["batch"].run(case["steps"])
        got = [sim.particles() for sim in state["sims"]]
        out = {k: np.concatenate([g[i] for g in got]) for i, k in enumerate("xvf")}
    elif case["kind"] == ROUND_TRIP:
        lib, sim, x, v, f = _lib.load(), state["sim"], state["x"], state["v"], state["f"]
        for _ in range(case["steps"]):
            _lib.check(lib.selm_set_particles(sim._h, len(x), _ptr(x), _ptr(v), None))
            sim.run(1)
            _read(sim, x, v, f)
        out = dict(x=x, v=v, f=f)
    else:
        sim = state["sim"]
        sim.run(case["steps"])
        if case["sample"]:
            state["analysis"].sample()
        out = dict(zip("xvf", sim.particles()))
        if case["field"]:
            out["u"] = sim.get_field()
        if case["sample"]:
            out["msd"] = state["analysis"].msd_sums()[0]
            out["sq"] = state["analysis"].structure()[0]
    return _in_form(out, case["form"])


def _in_form(out, form):
    kind = torch.float32 if form == "fused32" else torch.float64
    return {k: torch.as_tensor(a).to(kind) for k, a in out.items()}


def work(case):
    """Per step: the fluid state read and written, the monomers' x, v, f and
    mass read and x, v, f written; two real transforms of three fields, the
    spectral update, two 64-point stencils per monomer component."""
    total = dict(bytes=0.0, flops=0.0)
    for c in _members(case) if case["kind"] == BATCH else [case]:
        N, M = float(c["grid"]) ** 3, float(c["chains"] * c["length"])
        s = 4 if c["form"] == "fused32" else 8
        total["bytes"] += case["steps"] * (6 * N * s + M * (6 * 24 + 8))
        total["flops"] += case["steps"] * (15 * N * math.log2(N) + 40 * N + M * 3 * 64 * 4)
    return total


# ---------------------------------------------------------------- the same in 64 bits
def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors that hold 32-bit words."""
    mask = 0xFFFFFFFF
    k0, k1 = seed & mask, (seed >> 32) & mask
    c0, c1, c2, c3 = torch.broadcast_tensors(c0, c1, c2, c3)
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & mask) ^ c1 ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c3 ^ k1, p0 & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c0, c1, c2, c3


def _normals(q, d, step, seed):
    """Box-Muller pairs of the 52-bit uniforms of counter (q, d, step)."""
    word = lambda v: torch.full((1,), v, dtype=torch.int64, device=q.device)  # noqa: E731
    o = _philox(q, word(d), word(step & 0xFFFFFFFF), word(step >> 32), seed)
    u1, u2 = ((((a << 20) | (b >> 12)).double() + 0.5) * 2.0 ** -52 for a, b in (o[:2], o[2:]))
    r = torch.sqrt(-2.0 * torch.log(u1))
    return r * torch.cos(2.0 * math.pi * u2), r * torch.sin(2.0 * math.pi * u2)


class _Exact:
    """One simulation in FP64: u_hat is the fluid's state, u the field of it."""

    def __init__(self, par, x, v, mass, topo):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, k=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device=self.dev).to(k)  # noqa: E731
        self.p, self.n, self.lo, self.L = par, int(par.numMeshPtsPerDir[0]), par.box_lo, par.box_hi - par.box_lo
        self.dx = self.L / self.n
        self.x, self.v, self.m, self.topo = t(x), t(v), t(mass)[:, None], topo
        n, nh = self.n, self.n // 2 + 1
        self.types = t(topo.types, torch.int64)
        self.bonds, self.angles = t(topo.bonds, torch.int64).reshape(-1, 3), t(topo.angles, torch.int64).reshape(-1, 4)
        self.bc, self.ac = t(topo.bond_coeff), t(topo.angle_coeff)
        if topo.pair_style != "none":
            nt = topo.ntypes + 1
            self.pc = t(topo.pair_coeff).reshape(nt, nt, 3)
            # a pair of bonded monomers is left out; of the four-bead molecules every pair of one molecule
            self.apart = (lambda i, j: i // 4 != j // 4) if topo.angle_style != "none" else self._not_bonded
            self.follows = torch.zeros(len(x), dtype=torch.bool, device=self.dev)
            self.follows[self.bonds[:, 2]] = True  # bonded to the monomer before it
        # symbols: k along x last
        k = torch.arange(n, device=self.dev).double()
        cm, sn = -2.0 * torch.sin(math.pi * k / n) ** 2, torch.sin(2.0 * math.pi * k / n)
        view = [(1, 1, nh), (1, n, 1), (n, 1, 1)]
        d = [torch.complex(cm[: s[2]] if s[2] > 1 else cm, sn[: s[2]] if s[2] > 1 else sn).reshape(s) / self.dx for s in view]
        self.D = d
        self.Lk = sum(2.0 * (c[: s[2]] if s[2] > 1 else c).reshape(s) for c, s in zip((cm,) * 3, view)) / self.dx ** 2
        self.uh = torch.zeros((3, n, n, nh), dtype=torch.complex128, device=self.dev)
        self.u = torch.zeros((3, n, n, n), dtype=torch.float64, device=self.dev)
        self.step_no = 0
        self.f = self.forces()

    def _not_bonded(self, i, j):
        return ~(((j == i + 1) & self.follows[j]) | ((i == j + 1) & self.follows[i]))

    def near(self, d):
        return d - self.L * torch.round(d / self.L)

    # -- forces
    def forces(self):
        t, f = self.topo, torch.zeros_like(self.x)
        if len(self.bonds):
            ty, i, j = self.bonds.T
            c, d = self.bc[ty], self.near(self.x[i] - self.x[j])
            r2 = (d * d).sum(1)
            if t.bond_style == "harmonic":
                r = torch.sqrt(r2)
                s = -2.0 * c[:, 0] * (r - c[:, 1]) / r
            else:
                s = -c[:, 0] / torch.clamp(1.0 - r2 / c[:, 1] ** 2, min=0.1)
                s6 = (c[:, 3] ** 2 / r2) ** 3
                s = s + torch.where(r2 < 2.0 ** (1.0 / 3.0) * c[:, 3] ** 2, 48.0 * c[:, 2] * s6 * (s6 - 0.5) / r2, 0.0)
            f.index_add_(0, i, s[:, None] * d)
            f.index_add_(0, j, -s[:, None] * d)
        if len(self.angles):
            ty, i, j, k = self.angles.T
            a, b = self.near(self.x[i] - self.x[j]), self.near(self.x[k] - self.x[j])
            ra, rb = torch.linalg.norm(a, dim=1), torch.linalg.norm(b, dim=1)
            c = torch.clamp((a * b).sum(1) / (ra * rb), -1.0, 1.0)
            s = 1.0 / torch.clamp(torch.sqrt(1.0 - c * c), min=0.001)
            g = -2.0 * self.ac[ty, 0] * (torch.acos(c) - self.ac[ty, 1] * math.pi / 180.0) * s
            fa = (g * c / ra ** 2)[:, None] * a - (g / (ra * rb))[:, None] * b
            fb = (g * c / rb ** 2)[:, None] * b - (g / (ra * rb))[:, None] * a
            f.index_add_(0, i, fa)
            f.index_add_(0, k, fb)
            f.index_add_(0, j, -(fa + fb))
        if t.pair_style != "none":
            self.pairs(f)
        return f + torch.as_tensor(np.array(t.body_force, float), device=self.dev)

    def pairs(self, f):
        M, rc = len(self.x), float(self.pc[..., 2].max())
        all_ = torch.arange(M, device=self.dev)
        if M <= 2500:
            parts = [(all_[:, None].expand(M, M), all_[None, :].expand(M, M))]
        else:
            nc = int(self.L / rc)
            c = torch.clamp(((self.x - self.lo) / self.L * nc).long(), 0, nc - 1)
            flat = (c[:, 2] * nc + c[:, 1]) * nc + c[:, 0]
            order = torch.argsort(flat)
            count = torch.bincount(flat, minlength=nc ** 3)
            start = torch.cumsum(count, 0) - count
            slot = torch.empty_like(all_)
            slot[order] = all_ - start[flat[order]]
            table = torch.full((nc ** 3, int(count.max())), -1, dtype=torch.int64, device=self.dev)
            table[flat, slot] = all_
            parts = []
            for q in range(27):
                o = torch.tensor([q % 3 - 1, q // 3 % 3 - 1, q // 9 - 1], device=self.dev)
                e = torch.remainder(c + o, nc)
                j = table[(e[:, 2] * nc + e[:, 1]) * nc + e[:, 0]]
                parts.append((all_[:, None].expand_as(j), j))
        for i, j in parts:
            hit = (j >= 0) & (j != i)
            i, j = i[hit], j[hit]
            d = self.near(self.x[i] - self.x[j])
            r2 = (d * d).sum(1)
            c = self.pc[self.types[i], self.types[j]]
            hit = (r2 < c[:, 2] ** 2) & self.apart(i, j)
            i, d, r2, c = i[hit], d[hit], r2[hit], c[hit]
            s6 = (c[:, 1] ** 2 / r2) ** 3
            f.index_add_(0, i, (24.0 * c[:, 0] * s6 * (2.0 * s6 - 1.0) / r2)[:, None] * d)

    # -- coupling
    def stencil(self, d):
        """Flat cells [M, 64] and weights of component d's Peskin stencil."""
        g = (self.x - self.lo) / self.dx
        idx, wt = [], []
        for a in range(3):
            r = g[:, a] - (0.0 if a == d else 0.5)
            p = torch.floor(r)[:, None] - 1.0 + torch.arange(4, device=self.dev)
            q = torch.abs(r[:, None] - p)
            inner = (3.0 - 2.0 * q + torch.sqrt(torch.clamp(1.0 + 4.0 * q * (1.0 - q), min=0.0))) / 8.0
            outer = (5.0 - 2.0 * q - torch.sqrt(torch.clamp(-7.0 + 4.0 * q * (3.0 - q), min=0.0))) / 8.0
            idx.append(torch.remainder(p.long(), self.n))
            wt.append(torch.where(q < 1.0, inner, outer))
        cell = (idx[2][:, :, None, None] * self.n + idx[1][:, None, :, None]) * self.n + idx[0][:, None, None, :]
        w = wt[2][:, :, None, None] * wt[1][:, None, :, None] * wt[0][:, None, None, :]
        return cell.reshape(len(g), 64), w.reshape(len(g), 64)

    def gathered(self):
        return torch.stack([(self.u[d].reshape(-1)[c] * w).sum(1) for d in range(3) for c, w in [self.stencil(d)]], 1)

    def spread(self, t):
        g = torch.zeros_like(self.u)
        for d in range(3):
            c, w = self.stencil(d)
            g[d].view(-1).index_add_(0, c.reshape(-1), (t[:, d, None] * w).reshape(-1))
        return g

    # -- fluid
    def noise(self):
        """The thermal forcing's spectrum of this step, before its prefactor:
        variance lambda_h, Hermitian average on the x = 0 and Nyquist planes."""
        n, nh = self.n, self.n // 2 + 1
        q = torch.arange(n * n * nh, device=self.dev)
        amp = torch.sqrt(-self.Lk)
        k = torch.arange(n, device=self.dev)
        own = (2 * k) % n == 0
        selfc = own[:, None, None] & own[None, :, None] & own[None, None, :nh]
        full = self.p.noise_mode == "exact" or self.p.integrator == "quasi_steady"
        out = torch.empty_like(self.uh)
        for d in range(3):
            a, b = _normals(q, d, self.step_no, int(self.p.SELM_Seed))
            z = torch.complex(a, b).reshape(n, n, nh)
            z = torch.where(selfc, torch.complex(z.real, torch.zeros_like(z.real)), z * math.sqrt(0.5)) * amp
            for i in range(nh):
                if i == 0 or 2 * i == n:
                    m = z[:, :, i]
                    mirror = torch.roll(torch.flip(m, (0, 1)), (1, 1), (0, 1)).conj()
                    z[:, :, i] = torch.where(selfc[:, :, i], m, (m + mirror) * (math.sqrt(0.5) if full else 0.5))
            out[d] = z
        return out

    def project(self, w):
        """w - G (D . w) / L, the zero mode removed."""
        L = self.Lk.clone()
        L[0, 0, 0] = 1.0
        s = sum(self.D[d] * w[d] for d in range(3)) / L
        w = torch.stack([w[d] + self.D[d].conj() * s for d in range(3)])
        w[:, 0, 0, 0] = 0.0
        return w

    def to_field(self, wh):
        return torch.fft.irfftn(wh, s=(self.n,) * 3, dim=(1, 2, 3))

    def wrap(self, x):
        hi = self.lo + self.L
        return torch.where(x > hi, x - self.L, torch.where(x < self.lo, x + self.L, x))

    def step(self):
        p, N = self.p, float(self.n) ** 3
        self.step_no += 1
        hot = bool(p.flagStochasticDriving)
        kT = p.KB * p.T
        if p.integrator == "quasi_steady":
            Fh = torch.fft.rfftn(self.spread(self.f / self.dx ** 3), dim=(1, 2, 3))
            if hot:
                Fh += math.sqrt(2.0 * kT * p.mu * N / (p.dt * self.dx ** 3)) * self.noise()
            L = self.Lk.clone()
            L[0, 0, 0] = 1.0
            self.u = self.to_field(self.project(Fh) / (-p.mu * L))
            self.v = self.gathered()
            self.x = self.wrap(self.x + p.dt * self.v)
        else:
            ups = 12.0 * math.pi * self.dx * p.mu
            tf = -ups * (self.v - self.gathered()) * p.dt
            if hot:
                q = torch.arange(len(self.x), device=self.dev)
                z = torch.stack([_normals(q, 4 + d, self.step_no, int(p.SELM_Seed))[0] for d in range(3)], 1)
                tf = tf + math.sqrt(2.0 * kT * ups * p.dt) * z
            Fh = torch.fft.rfftn(self.spread(-tf), dim=(1, 2, 3))
            if hot:
                Fh += math.sqrt(2.0 * kT * p.dt * p.mu / N) * N * self.noise()
            new_x = self.wrap(self.x + p.dt * self.v)
            self.v = self.v + (tf + p.dt * self.f) / self.m
            self.x = new_x
            self.uh = self.project(self.uh * (1.0 + p.mu * p.dt * self.Lk / p.rho) + Fh / p.rho)
            self.u = self.to_field(self.uh)
        self.f = self.forces()


def _exact_run(system, steps):
    sim = _Exact(*system)
    for _ in range(WARM):
        sim.step()
    before = sim.x.clone()
    for _ in range(steps):
        sim.step()
    return sim, before


def exact(case, seed):
    if case["kind"] == BATCH:
        got = [_exact_run(_system(m, 1000 * seed + k), case["steps"])[0] for k, m in enumerate(_members(case))]
        return {k: torch.cat([getattr(g, k) for g in got]).cpu() for k in "xvf"}
    sim, before = _exact_run(_system(case, seed), case["steps"])
    out = {k: getattr(sim, k).cpu() for k in "xvf"}
    if case["field"] and case["kind"] == RUN:
        out["u"] = sim.u.cpu()
    if case["sample"]:
        # frames are float32, as a trajectory's
        d = sim.near((sim.x.float() - before.float()).double())
        out["msd"] = torch.zeros((NLAG, 3), dtype=torch.float64)
        out["msd"][0] = (d * d).sum(0).cpu()
        sq = []
        for x in (before, sim.x):
            phase = 2.0 * math.pi / sim.L * x @ torch.tensor(QVEC, dtype=torch.float64, device=sim.dev).T
            sq.append((torch.cos(phase).sum(0) ** 2 + torch.sin(phase).sum(0) ** 2) / len(x))
        out["sq"] = ((sq[0] + sq[1]) / 2.0).cpu()
    return out
