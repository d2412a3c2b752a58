"""Performance cases of the sLLG step.

What a program built on this library spends its time in is `Handle.step` with the reads between
the steps, so a case is a lattice with its interactions, an arithmetic form and integrator, and
one pass of the program's inner loop: advance a number of steps, read the magnetisation, read the
spins into a page-locked buffer that the program keeps.  The lattices are those of the bench and
the tests (sc, BCT-2, J1+J2 film, uneven sc replicas; exchange in CSR, DIA or folded into the
FFT; dipole by FFT), at those sizes, smaller ones and ragged ones.

`exact` restates the same pass in FP64 with plain torch: the bonds applied as shifted copies of the
lattice, the long-range field by torch.fft on a zero-padded mesh, the thermal normals from the
published Philox4x32-10 and Box-Muller.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(REPO, "gpu-atomistic-code_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import asd_b200 as A  # noqa: E402
import asd_lattice as LT  # noqa: E402

FORMS = {"fp32": A.FP32, "fused64": A.FP64_FUSED, "plain64": A.FP64_PLAIN}
INTEGRATORS = {"heun": A.HEUN, "rk4": A.RK4, "rk5": A.RK5}
PULSE = (0.1, 2e-14, 1e-14)        # site-field pulse: amplitude [T], centre [s], width [s]


def case(kind, dim, steps, name=None, form="fp32", integrator="heun", exch="csr", periodic=True, dipole=False, T=0.0,
         dt=1e-16, tune=False, loop="steps", nrep=1, lattice_seed=0):
    """`dim`: cells per axis (replicas: the range of the edges).  `loop`: "steps" advances them in
    one call, "drive" sets the applied field and reads the magnetisation at every step, "sample"
    accumulates M(T) statistics every 10 steps.  `tune`: the launch shape by the autotuner."""
    c = dict(kind=kind, nx=dim[0], ny=dim[1], nz=dim[2], steps=steps, form=form, integrator=integrator, exch=exch,
             periodic=periodic, dipole=dipole, T=T, dt=dt, tune=tune, loop=loop, nrep=nrep, lattice_seed=lattice_seed)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest lattice in use (config 0): a trajectory at 300 K, bound by launches
        case("sc", (16, 16, 16), 192, "sc16_heat", T=300.0),
        # a host driver (field ramp): applied field in, one step, magnetisation out, every step
        case("sc", (24, 24, 24), 64, "sc24_field_drive", T=100.0, loop="drive"),
        # the bench's BCT-2 lattice: 26 neighbours, full tensors, 300 K
        case("bct2", (64, 64, 64), 64, "bct2_64", T=300.0, tune=True),
        # the same exchange given as DIA, on a ragged lattice of ordinary size, untuned
        case("bct2", (37, 29, 23), 128, "bct2_37x29x23_dia", exch="dia", T=300.0),
        # the bench's default: a million spins, exchange and the dipole field every step
        case("sc", (128, 128, 64), 60, "sc128x128x64_dipole", periodic=False, dipole=True, tune=True),
        # a sample of arbitrary edges with the dipole field at finite temperature
        case("sc", (90, 75, 41), 40, "sc90x75x41_dipole", periodic=False, dipole=True, T=100.0),
        # spin waves: J1+J2 film in DIA, dipole, site-field pulse, RK4
        case("film", (256, 256, 4), 40, "film256x256x4_rk4", integrator="rk4", exch="dia", dipole=True, dt=5e-16),
        # exchange folded into the FFT field, evaluated at every stage
        case("sc_fft", (64, 64, 64), 40, "sc64_fft", exch="fft", periodic=False, dipole=True),
        # M(T): uneven replicas at their own temperatures, statistics every 10 steps
        case("replicas", (16, 64, 1), 50, "replicas24_mvt", T=125.0, loop="sample", nrep=24, lattice_seed=4),
        # a large periodic lattice at finite temperature, exchange only
        case("sc", (128, 128, 128), 50, "sc128_heat", T=300.0, tune=True),
        # the fused FP64 form with the dipole field
        case("sc", (64, 64, 32), 60, "sc64x64x32_dipole_fused64", form="fused64", periodic=False, dipole=True),
        # the FP64 plain form: the runs that others are checked against
        case("bct2", (24, 24, 24), 32, "bct2_24_plain64", form="plain64", T=300.0),
    ]


def draw(rng):
    """A case of the same ranges: edges log-uniform, odd ones included."""
    def edge(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi, most):
        while True:
            d = [edge(lo, hi) for _ in range(3)]
            if d[0] * d[1] * d[2] <= most:
                return d

    def steps_for(n, cost):
        return max(4, min(128, int(4e7 / (cost * n))))

    form = rng.choice(["fp32"] * 6 + ["fused64", "plain64"])
    integ = rng.choice(["heun", "heun", "heun", "rk4", "rk5"])
    T = rng.choice([0.0, 50.0, 100.0, 300.0])
    tune = rng.random() < 0.5
    slow = {"fp32": 1, "fused64": 3, "plain64": 8}[form]
    stages = {"heun": 1, "rk4": 2, "rk5": 3}[integ]
    kind = rng.choice(["sc", "sc", "sc_dipole", "sc_dipole", "bct2", "bct2_dia", "film", "sc_fft", "replicas"])
    if kind == "sc":
        d = dims(8, 128, 1 << 20)
        loop = rng.choice(["steps", "steps", "drive"])
        return case("sc", d, steps_for(d[0] * d[1] * d[2], stages * slow), form=form, integrator=integ,
                    periodic=rng.random() < 0.7, T=T, tune=tune, loop=loop)
    if kind == "sc_dipole":
        d = dims(8, 128, 1 << 18)
        return case("sc", d, steps_for(d[0] * d[1] * d[2], 4 * stages * slow), form=form, integrator=integ, periodic=False,
                    dipole=True, T=T, tune=tune)
    if kind in ("bct2", "bct2_dia"):
        d = dims(6, 64, 1 << 16)
        return case("bct2", d, steps_for(2 * d[0] * d[1] * d[2], 2 * stages * slow), form=form, integrator=integ,
                    exch="dia" if kind == "bct2_dia" else "csr", T=T, tune=tune)
    if kind == "film":
        d = [edge(48, 256), edge(48, 256), rng.randint(1, 6)]
        return case("film", d, steps_for(d[0] * d[1] * d[2], 6 * slow), form=form, integrator="rk4", exch="dia",
                    dipole=rng.random() < 0.7, dt=5e-16, tune=tune)
    if kind == "sc_fft":
        d = dims(8, 72, 1 << 17)
        return case("sc_fft", d, steps_for(d[0] * d[1] * d[2], 8 * slow), form=form, integrator="heun", exch="fft",
                    periodic=False, dipole=True, T=T)
    nrep = rng.randint(4, 24)
    lo = edge(8, 24)
    return case("replicas", (lo, rng.randint(lo, 48), 1), rng.choice([20, 30, 40]), form=form, T=125.0, tune=tune,
                loop="sample", nrep=nrep, lattice_seed=rng.randrange(1000))


# ---------------------------------------------------------------- the program's side
def replica_edges(c):
    return [int(v) for v in np.random.default_rng(c["lattice_seed"]).integers(c["nx"], c["ny"] + 1, c["nrep"])]


def replica_temperatures(c):
    return [float(v) for v in np.linspace(0.0, c["T"], c["nrep"])]


@functools.lru_cache(maxsize=1)
def systems(key):
    """The lattices of a case with their interactions (the same for every run of a program)."""
    c = dict(key)
    dim = (c["nx"], c["ny"], c["nz"])
    pbc = (1, 1, 1) if c["periodic"] else (0, 0, 0)
    if c["kind"] == "sc":
        return [LT.sc_ferromagnet(dim, pbc=pbc, T=c["T"], exch=c["exch"], dipole=c["dipole"])]
    if c["kind"] == "bct2":
        return [LT.bct2_antiferromagnet(dim, layout=c["exch"], T=c["T"])]
    if c["kind"] == "film":
        return [LT.film_dia(*dim, dipole=c["dipole"])]
    if c["kind"] == "sc_fft":
        return [LT.sc_fft(dim, T=c["T"])]
    return [LT.sc_ferromagnet(e, T=t, stream=r)
            for r, (e, t) in enumerate(zip(replica_edges(c), replica_temperatures(c)))]


def spin_count(c):
    if c["kind"] == "replicas":
        return sum(e ** 3 for e in replica_edges(c))
    return c["nx"] * c["ny"] * c["nz"] * (2 if c["kind"] == "bct2" else 1)


def initial_spins(c, seed):
    """Partly ordered along z (the sublattices of BCT-2 against each other); for the spin-wave
    film, up with a random tilt of a few degrees."""
    rng = np.random.default_rng(seed)
    n = spin_count(c)
    v = rng.standard_normal((n, 3))
    if c["kind"] == "film":
        v *= 0.05
        v[:, 2] = 1.0
    elif c["kind"] == "bct2":
        v[0::2, 2] += 1.0
        v[1::2, 2] -= 1.0
    else:
        v[:, 2] += 1.0
    return v / np.sqrt((v * v).sum(axis=1, keepdims=True))


def noise_seed(seed):
    return 1 + int(seed) % 1000003


def drive_field(k):
    """The field ramp of the drive loop at its k-th step [T]."""
    return (0.05 * math.sin(0.1 * k), 0.0, 0.02 * k)


def prepare(c, seed):
    flags = (A.FLAG_COMPENSATED if c["form"] == "fp32" else 0) | (A.FLAG_AUTOTUNE if c["tune"] else 0)
    p = A.RunParams(integrator=INTEGRATORS[c["integrator"]], precision=FORMS[c["form"]], dt=c["dt"],
                    seed=noise_seed(seed), flags=flags)
    h = A.Handle(p, systems(tuple(sorted(c.items()))))
    if c["kind"] == "film":
        h.set_site_field_pulse(*PULSE)
    h.set_spins(initial_spins(c, seed))
    nmag = h.nrep * h.nsub * 3
    record = np.float64 if c["form"] == "plain64" else np.float32     # what the program keeps of the means
    return {"handle": h, "record": record, "loop": c["loop"], "steps": c["steps"],
            "spins": torch.empty(3 * h.n, dtype=torch.float64, pin_memory=True).numpy(),
            "mag": torch.empty(nmag, dtype=torch.float64, pin_memory=True).numpy(),
            "series": np.zeros((c["steps"], nmag), dtype=record)}


def run(state):
    h = state["handle"]
    if state["loop"] == "drive":
        for k in range(state["steps"]):
            h.set_applied(drive_field(k))
            h.step(1)
            state["series"][k] = h.magnetisation(state["mag"]).reshape(-1)
        return {"spins": h.get_spins(state["spins"]), "magnetisation": state["series"]}
    if state["loop"] == "sample":
        for k in range(0, state["steps"], 10):
            h.step(min(10, state["steps"] - k))
            h.sample_magnetisation()
        stats = h.magnetisation_stats()[..., 1]
        h.reset_magnetisation_stats()
        return {"spins": h.get_spins(state["spins"]), "mean": stats.astype(state["record"])}
    h.step(state["steps"])
    return {"magnetisation": h.magnetisation(state["mag"]).astype(state["record"]), "spins": h.get_spins(state["spins"])}


def work(c):
    """Per stage the spins come in and the new ones go out once (FP32: hi + lo at the step's
    ends); a long-range field adds its mesh sites in and out and one octant of N_k, and the
    pruned transforms of three components there and back."""
    n, b = spin_count(c), 4 if c["form"] == "fp32" else 8
    stages = {"heun": 2, "rk4": 4, "rk5": 6}[c["integrator"]]
    bonds = {"sc": 6 * 6, "bct2": 26 * 18, "film": 18 * 6, "sc_fft": 0, "replicas": 6 * 6}[c["kind"]]
    nbytes = n * (stages * 6 * b + (24 if b == 4 else 0))
    flops = n * stages * (bonds + 80)
    if c["dipole"]:
        evals = stages if c["kind"] == "sc_fft" else 1
        nbytes += evals * (24 * n + 6 * 4 * (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1))
        flops += evals * 6 * 5 * 2.0 * n * math.log2(8.0 * n)
    return {"bytes": float(c["steps"] * nbytes + 24 * n), "flops": float(c["steps"] * flops)}


# ---------------------------------------------------------------- the same pass in FP64
MUB, KB, GYRO = 9.27e-24, 1.38e-23, 1.76e11
SC = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1)]
FACES = [(a, b, 0) for a in (1, -1) for b in (1, -1)] + [(a, 0, b) for a in (1, -1) for b in (1, -1)] + \
        [(0, a, b) for a in (1, -1) for b in (1, -1)]


def bct2_bonds():
    """(atom, neighbour atom, cell offset, tensor [J]) of the BCT-2 lattice's seeded tensors."""
    rng = np.random.default_rng(2)
    tensors = {}
    for key in [(0, 1, 1), (0, 0, 2), (1, 1, 2), (0, 0, 3), (1, 1, 3), (0, 0, 4), (1, 1, 4)]:
        d = rng.uniform(-2e-21, 1e-21, 3)
        D = rng.uniform(-1.0, 1.0, 3) * 0.05 * np.abs(d).mean()
        tensors[key] = np.diag(d) + np.array([[0, D[2], -D[1]], [-D[2], 0, D[0]], [D[1], -D[0], 0]])
    out = []
    for v in [(a, b, c) for a in (0, -1) for b in (0, -1) for c in (0, -1)]:
        out.append((0, 1, v, tensors[(0, 1, 1)]))
        out.append((1, 0, tuple(-x for x in v), tensors[(0, 1, 1)].T))
    for shell, vecs in ((2, SC[4:]), (3, SC[:4]), (4, FACES)):
        for a in (0, 1):
            for v in vecs:
                J = tensors[(a, a, shell)]
                out.append((a, a, v, J if v > (0, 0, 0) else J.T))
    return out


class Lattice:
    """One lattice in FP64: spins [x, y, z, atom, 3] on `dev`."""

    def __init__(self, c, dim, T, stream, seed, spins, dev):
        self.dev, self.dim, self.T, self.stream, self.seed = dev, tuple(dim), T, stream, seed
        kind, self.kind = c["kind"], c["kind"]
        self.mu, self.lam, self.k1u = 1.5, 0.1, 1e-23
        self.pbc, self.na = ((1, 1, 1) if c["periodic"] else (0, 0, 0)), 1
        J = 1e-21
        bonds = [(0, 0, v, J * np.eye(3)) for v in SC]
        if kind == "bct2":
            self.lam, self.k1u, self.na, self.pbc, bonds = 0.01, -1e-23, 2, (1, 1, 1), bct2_bonds()
        elif kind == "film":
            self.lam, self.k1u, self.pbc = 1e-4, 0.0, (1, 1, 0)
            bonds += [(0, 0, v, -0.2 * J * np.eye(3)) for v in FACES]
        elif kind == "replicas":
            self.pbc = (1, 1, 1)
        elif kind == "sc_fft":
            self.pbc = (0, 0, 0)
        self.bonds = [(a, t, v, torch.tensor(Jm / (self.mu * MUB), device=dev)) for a, t, v, Jm in bonds]
        self.S = torch.tensor(spins, device=dev).reshape(*self.dim, self.na, 3)
        self.dt, self.rdt, self.integrator = c["dt"], c["dt"] * GYRO, c["integrator"]
        self.sigma = math.sqrt(2.0 * KB * self.lam / (self.mu * MUB * self.dt * GYRO)) * math.sqrt(T)
        self.aniso = 2.0 * self.k1u / (self.mu * MUB)
        self.every_stage = kind == "sc_fft"
        self.nk = self.kernel() if c["dipole"] else None
        self.t, self.applied = 0, torch.zeros(3, dtype=torch.float64, device=dev)
        self.site = None
        if kind == "film":
            x = (torch.arange(self.dim[0], dtype=torch.float64, device=dev) - self.dim[0] / 2) / 16.0
            self.site = torch.zeros(*self.dim, 1, 3, dtype=torch.float64, device=dev)
            self.site[..., 0] = torch.sinc(x)[:, None, None, None]

    def kernel(self):
        """Transforms of the point-dipole tensor on the doubled mesh (6 components)."""
        m = [2 * d for d in self.dim]
        ax = []
        for d in self.dim:
            i = torch.arange(2 * d, device=self.dev)
            ax.append(torch.where(i > d, i - 2 * d, i).double() * 3e-10)
        r = torch.meshgrid(*ax, indexing="ij")
        r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
        r2[0, 0, 0] = 1.0
        out = {}
        for a in range(3):
            for b in range(a, 3):
                g = 1e-7 * MUB * self.mu * (3.0 * r[a] * r[b] / r2 - (1.0 if a == b else 0.0)) * r2 ** -1.5
                g[0, 0, 0] = 0.0
                for k in range(3):                    # no two spins are half a mesh apart
                    g.select(k, self.dim[k]).zero_()
                out[a, b] = torch.fft.rfftn(g)
        self.mesh = m
        return out

    def long_range(self, S):
        F = [torch.fft.rfftn(S[..., 0, a], s=self.mesh) for a in range(3)]
        d = self.dim
        H = torch.empty_like(S)
        for a in range(3):
            k = sum(self.nk[min(a, b), max(a, b)] * F[b] for b in range(3))
            H[..., 0, a] = torch.fft.irfftn(k, s=self.mesh)[: d[0], : d[1], : d[2]]
        return H

    def exchange(self, S):
        H = torch.zeros_like(S)
        for a, t, v, J in self.bonds:
            G = torch.roll(S[..., t, :], shifts=[-x for x in v], dims=(0, 1, 2))
            for k in range(3):
                if v[k] and not self.pbc[k]:
                    edge = slice(self.dim[k] - v[k], None) if v[k] > 0 else slice(0, -v[k])
                    G[(slice(None),) * k + (edge,)] = 0.0
            H[..., a, :] += G @ J.T
        return H

    def normals(self):
        """Philox4x32-10 (counter: spin, step, stream; key: seed), then Box-Muller."""
        n = self.S[..., 0].numel()
        M = 0xFFFFFFFF
        c = [torch.arange(n, device=self.dev), torch.full((n,), self.t & M, device=self.dev),
             torch.zeros(n, dtype=torch.int64, device=self.dev), torch.full((n,), self.stream, device=self.dev)]
        k0, k1 = self.seed & M, self.seed >> 32
        for _ in range(10):
            p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
            c = [(p1 >> 32 & M) ^ c[1] ^ k0, p1 & M, (p0 >> 32 & M) ^ c[3] ^ k1, p0 & M]
            k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
        u = [(x.double() + 0.5) * 2.0 ** -32 for x in c]
        r0, r2 = (torch.sqrt(-2.0 * torch.log(u[k])) for k in (0, 2))
        a1, a3 = 2 * math.pi * u[1], 2 * math.pi * u[3]
        return torch.stack([r0 * torch.cos(a1), r0 * torch.sin(a1), r2 * torch.cos(a3)], dim=1).reshape(self.S.shape)

    def torque(self, S, extra, lr):
        H = extra + self.aniso * S * torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device=self.dev)
        H = H + self.exchange(S)
        if lr is not None:
            H = H + lr
        a = torch.linalg.cross(S, H)
        return (a + self.lam * torch.linalg.cross(S, a)) * (-1.0 / (1.0 + self.lam ** 2))

    def step(self):
        S = self.S
        unit = lambda v: v / v.norm(dim=-1, keepdim=True)  # noqa: E731
        extra = self.applied.expand_as(S)
        if self.T > 0:
            extra = extra + self.sigma * self.normals()
        if self.site is not None:
            amp, t0, sg = PULSE
            extra = extra + self.site * (amp * math.exp(-0.5 * ((self.t * self.dt - t0) / sg) ** 2))
        held = self.long_range(S) if self.nk and not self.every_stage else None

        def f(v):
            return self.torque(v, extra, self.long_range(v) if self.every_stage else held)

        if self.integrator == "heun":
            f0 = f(S)
            self.S = unit(S + 0.5 * self.rdt * (f0 + f(unit(S + self.rdt * f0))))
        else:
            if self.integrator == "rk4":
                B, C = [[0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6]
            else:                                      # Cash-Karp
                B = [[1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
                     [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
                C = [37 / 378, 0.0, 250 / 621, 125 / 594, 0.0, 512 / 1771]
            k = [self.rdt * f(S)]
            for row in B:
                k.append(self.rdt * f(unit(S + sum(w * q for w, q in zip(row, k)))))
            self.S = unit(S + sum(w * q for w, q in zip(C, k)))
        self.t += 1

    def advance(self, steps):
        for _ in range(steps):
            self.step()

    def magnetisation(self):
        return self.S.mean(dim=(0, 1, 2))


def exact(c, seed):
    if c["integrator"] != "heun" and c["kind"] == "sc_fft":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    S0 = initial_spins(c, seed)
    if c["kind"] == "replicas":
        lats, off = [], 0
        for r, (e, t) in enumerate(zip(replica_edges(c), replica_temperatures(c))):
            lats.append(Lattice(c, (e, e, e), t, r, noise_seed(seed), S0[off:off + e ** 3], dev))
            off += e ** 3
    else:
        lats = [Lattice(c, (c["nx"], c["ny"], c["nz"]), c["T"], 0, noise_seed(seed), S0, dev)]
    spins = lambda: torch.cat([q.S.reshape(-1, 3) for q in lats]).cpu().numpy()  # noqa: E731
    if c["loop"] == "drive":
        series = []
        for k in range(c["steps"]):
            lats[0].applied = torch.tensor(drive_field(k), dtype=torch.float64, device=dev)
            lats[0].step()
            series.append(lats[0].magnetisation().reshape(-1))
        return {"spins": spins(), "magnetisation": torch.stack(series).cpu().numpy()}
    if c["loop"] == "sample":
        means = []
        for q in lats:
            m = []
            for k in range(0, c["steps"], 10):
                q.advance(min(10, c["steps"] - k))
                m.append(q.magnetisation().norm(dim=-1))
            means.append(torch.stack(m).mean(dim=0))
        return {"spins": spins(), "mean": torch.stack(means).cpu().numpy()}
    for q in lats:
        q.advance(c["steps"])
    return {"magnetisation": torch.stack([q.magnetisation() for q in lats]).cpu().numpy(), "spins": spins()}
