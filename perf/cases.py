"""The work whose time is measured: one pass per case through the public
entry points (``System`` and ``Batch`` of the package), as a program that uses
the library calls them, over the range of sizes it is used for.

Kinds of case:
  md           a state set from device arrays, a run of MD steps, the state
               back: a production run between two dumps;
  host_loop    one MD step per call with the state on the host, page-locked
               (``step_io``): a host program that owns the state;
  ensemble     many independent replicas in one batch;
  observables  the estimators a run logs every `sfreq` steps;
  exchange     V_B, its estimators and the exterior spring forces alone.

Systems, in the units of the library (Hartree atomic units):
  trap    bosons of 1 Da in a 3 meV harmonic trap, no interaction;
  pair    the same trap with a 1 meV harmonic interaction of every pair;
  liquid  He-4 at 0.0218 A^-3 in a periodic box, Aziz interaction;
  dipole  2D bosons with an r^-3 interaction (no cutoff) in a 1 meV trap.

``exact`` restates the same step in plain torch, in 64 bits.
"""
import importlib
import math

import numpy as np
import torch

pk = importlib.import_module("pimd-b_gb300")

ANG = 1.8897261
KELVIN = 3.1668152e-06
MEV = 0.036749326e-3
DALTON = 1822.8885
FS = 4.1341373e16 * 1e-15
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


def listed():
    return [
        # the smallest call: a handful of trapped bosons, the host holding
        # the state and calling step by step; launches and latency only
        dict(name="host-loop-5x8", kind="host_loop", system="trap", N=5, P=8, T=1.0, steps=1),
        # trapped bosons, velocity Verlet and Langevin: the textbook run
        dict(name="trap-16x32", kind="md", system="trap", N=16, P=32, T=1.0, steps=50),
        # distinguishable particles, normal modes of a bead count that is no
        # power of two, Nose-Hoover chains per particle
        dict(name="chain-61x20", kind="md", system="pair", N=61, P=20, T=2.0, steps=20, bosonic=False,
             propagator="normal_modes", thermostat="nose_hoover_np"),
        # liquid He-4, the headline system: normal modes with their thermostat
        dict(name="liquid-256x64", kind="md", system="liquid", N=256, P=64, T=1.5, steps=20,
             propagator="normal_modes", nmthermostat=True),
        # the same with the state on the host at every step
        dict(name="host-loop-256x64", kind="host_loop", system="liquid", N=256, P=64, T=1.5, steps=1,
             propagator="normal_modes", nmthermostat=True),
        # its estimators, logged every few steps
        dict(name="observables-256x64", kind="observables", system="liquid", N=256, P=64, T=1.5),
        # long-range interaction: every pair of every bead
        dict(name="dipole-1024x32", kind="md", system="dipole", N=1024, P=32, T=2.0, steps=4),
        # the largest liquid: short cutoff, cell lists, mixed precision
        dict(name="liquid-4096x128-mixed", kind="md", system="liquid", N=4096, P=128, T=1.0, steps=4,
             propagator="normal_modes", precision="mixed"),
        # a degenerate gas: long exchange cycles, evaluated on their own
        dict(name="exchange-777x16", kind="exchange", system="trap", N=777, P=16, T=1.0),
        # the sum over permutations, for small systems
        dict(name="factorial-10x8", kind="md", system="trap", N=10, P=8, T=1.0, steps=1, exchange="factorial"),
        # the ensemble workload in mixed precision
        dict(name="ensemble-512-mixed", kind="ensemble", system="pair", N=128, replicas=512, steps=25,
             precision="mixed"),
        # a small ensemble in FP64
        dict(name="ensemble-61-fp64", kind="ensemble", system="pair", N=100, replicas=61, steps=20,
             precision="fp64"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["trap", "chain", "liquid", "liquid", "dipole", "factorial", "host_loop", "observables",
                       "exchange", "ensemble", "ensemble"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    T = round(rng.uniform(0.5, 4.0), 3)
    if kind == "trap":
        return dict(kind="md", system="trap", N=log(3, 400), P=log(4, 96), T=T, steps=rng.randint(10, 40),
                    nmthermostat=rng.random() < 0.3)
    if kind == "chain":
        return dict(kind="md", system="pair", N=log(8, 200), P=log(5, 40), T=T, steps=rng.randint(5, 20),
                    bosonic=False, propagator=rng.choice(["normal_modes", "cartesian"]), precision=precision,
                    thermostat=rng.choice(["langevin", "none", "nose_hoover_np", "nose_hoover_np_dim"]))
    if kind == "liquid":
        P = log(8, 128)
        N = min(log(32, 4096), 4096 * 128 // P)
        return dict(kind="md", system="liquid", N=N, P=P, T=T, steps=rng.randint(2, 4), precision=precision,
                    propagator=rng.choice(["normal_modes", "cartesian"]), nmthermostat=rng.random() < 0.5)
    if kind == "dipole":
        return dict(kind="md", system="dipole", N=log(50, 1024), P=log(4, 32), T=T, steps=rng.randint(2, 4),
                    precision=precision)
    if kind == "factorial":
        return dict(kind="md", system="trap", N=rng.randint(3, 11), P=log(4, 32), T=T, steps=1,
                    exchange="factorial")
    if kind == "host_loop":
        liquid = rng.random() < 0.5
        return dict(kind="host_loop", system="liquid" if liquid else "trap", N=log(32 if liquid else 3, 300),
                    P=log(4, 64), T=T, steps=1, propagator="normal_modes" if liquid else "cartesian",
                    nmthermostat=liquid)
    if kind == "observables":
        return dict(kind="observables", system=rng.choice(["liquid", "liquid", "dipole"]), N=log(32, 256),
                    P=log(8, 64), T=T)
    if kind == "exchange":
        return dict(kind="exchange", system=rng.choice(["trap", "liquid"]), N=log(32, 900), P=log(4, 32), T=T)
    return dict(kind="ensemble", system="pair", N=log(8, 128), replicas=log(16, 512), steps=rng.randint(2, 4),
                precision=rng.choice(["mixed", "fp64"]))


# ------------------------------------------------------------------- set-up

def _system(case, N, P, T, seed, replica=0):
    """Parameters of one system; the keys of make_config."""
    c = dict(ndim=3, natoms=N, nbeads=P, bosonic=int(case.get("bosonic", True)), pbc=0, fixcom=1,
             propagator=case.get("propagator", "cartesian"), thermostat=case.get("thermostat", "langevin"),
             nmthermostat=int(case.get("nmthermostat", False)), precision=case.get("precision", "fp64"),
             temperature=T * KELVIN, mass=1.0 * DALTON, size=10.0 * ANG, dt=1.0 * FS, gamma=-1.0, ext_kind="free",
             ext_params=(0.0, 0.0, 0.0), int_kind="free", int_params=(0.0, 0.0, 0.0), cutoff=-1.0 * ANG,
             seed=12345 + seed, replica=replica, exchange=case.get("exchange", "feldman_hirshberg"), nchains=4)
    kind = case["system"]
    if kind in ("trap", "pair"):
        c.update(ext_kind="harmonic", ext_params=(3.0 * MEV, 0.0, 0.0))
        if kind == "pair":
            c.update(int_kind="harmonic", int_params=(1.0 * MEV, 0.0, 0.0))
    elif kind == "dipole":
        c.update(ndim=2, size=60.0 * ANG * math.sqrt(N / 1024.0), ext_kind="harmonic",
                 ext_params=(1.0 * MEV, 0.0, 0.0), int_kind="dipole", int_params=(2.4799673e-4, 0.0, 0.0))
    else:
        box = (N / 0.0218) ** (1.0 / 3.0)
        # half the box for the small liquids, the usual 7 A (cell lists) for the large ones
        cut = 0.5 * box if N < 1000 else 7.0
        c.update(mass=4.0026 * DALTON, dt=2.0 * FS, pbc=1, size=box * ANG, int_kind="aziz", cutoff=cut * ANG)
    return c


def _initial(case, c, gen):
    """Positions and momenta [bead][particle][axis] on the device."""
    N, P, D, L = c["natoms"], c["nbeads"], c["ndim"], c["size"]
    if case["system"] in ("trap", "pair"):
        centre = (torch.rand(N, D, dtype=F64, device=DEV, generator=gen) - 0.5) * L
    else:  # a filled grid of cells, the particles near their cells' centres
        n = max(int(math.ceil(N ** (1.0 / D) - 1e-7)), 1)
        k = torch.arange(N, device=DEV)
        cell = torch.stack([(k // n ** (D - 1 - a)) % n for a in range(D)], 1).to(F64)
        centre = (cell + 0.5) * (L / n) - 0.5 * L
        centre = centre + 0.05 * ANG * torch.randn(N, D, dtype=F64, device=DEV, generator=gen)
    x = centre[None] + 0.05 * ANG * torch.randn(P, N, D, dtype=F64, device=DEV, generator=gen)
    # Maxwell-Boltzmann at the ring polymer's temperature
    p = math.sqrt(c["mass"] * c["temperature"] * P) * torch.randn(P, N, D, dtype=F64, device=DEV, generator=gen)
    return x, p


def _inputs(case, seed):
    """[(parameters, x, p)] of every system of the case."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    if case["kind"] != "ensemble":
        c = _system(case, case["N"], case["P"], case["T"], seed % 100000)
        return [(c, *_initial(case, c, gen))]
    rng = np.random.default_rng(12345)  # the ensemble's make-up; the states come from the seed
    out = []
    for r in range(case["replicas"]):
        N, P = int(rng.integers(max(3, case["N"] // 16), case["N"] + 1)), int(rng.choice([16, 32, 64]))
        T = float(rng.uniform(0.5, 4.0))
        c = _system(case, N, P, T, seed % 100000, r)
        out.append((c, *_initial(case, c, gen)))
    return out


def prepare(case, seed):
    systems = _inputs(case, seed)
    st = dict(case=case)
    if case["kind"] == "ensemble":
        # page-locked host arrays, the replicas' one after the other
        st["x"], st["p"] = (torch.cat([s[k].reshape(-1) for s in systems]).cpu().pin_memory().numpy() for k in (1, 2))
        st["out"] = [torch.empty(st["x"].shape, dtype=F64).pin_memory() for _ in range(3)]
        st["batch"] = pk.Batch([pk.make_config(**s[0]) for s in systems])
        return st
    c, x, p = systems[0]
    st["sys"] = pk.System(pk.make_config(**c))
    if case["kind"] == "host_loop":
        st["in"] = [x.cpu().pin_memory(), p.cpu().pin_memory()]
        st["out"] = [torch.empty(x.shape, dtype=F64).pin_memory() for _ in range(3)]
    else:
        st["in"] = [x.contiguous(), p.contiguous()]
        st["out"] = [torch.empty_like(x) for _ in range(3)]
    return st


def run(st):
    case = st["case"]
    if case["kind"] == "ensemble":
        b = st["batch"]
        b.set_states(st["x"], st["p"])
        b.step(case["steps"])
        # into arrays the program keeps: the C entry that Batch.get_states wraps
        b._c(pk.lib().pimdb_batch_get_states(b._b, *(pk.C.c_void_p(t.data_ptr()) for t in st["out"])))
        return st["out"]
    s = st["sys"]
    ins = [t.data_ptr() for t in st["in"]]
    outs = [t.data_ptr() for t in st["out"]]
    if case["kind"] == "host_loop":
        s.step_io_ptr(*ins, case["steps"], *outs)
        return st["out"]
    s.set_state_ptr(*ins, device=True)
    if case["kind"] == "md":
        s.step(case["steps"])
        s.get_state_ptr(*outs, device=True)
        return st["out"]
    got = s.observables() if case["kind"] == "observables" else s.exchange()
    return {k: np.float64(v) if isinstance(v, float) else v for k, v in got.items()}


def work(case):
    """Bytes: the state in and out once (the results alone for the
    estimators).  Operations: every pair of every bead once (with a cutoff,
    those inside it) at the cost of its force, a bead's springs and its update
    about 60 per particle and step, and the exchange's 19 N^2."""
    D = 2 if case["system"] == "dipole" else 3
    steps = case.get("steps", 1)
    if case["kind"] == "ensemble":
        # the mean over the replicas' sizes
        N2, N, P, R = case["N"] ** 2 / 3.0, case["N"] / 2.0, 112.0 / 3.0, case["replicas"]
    else:
        N, P, R = case["N"], case["P"], 1
        N2 = N * N
    pairs = 0.5 * N2
    per = {"trap": 0.0, "pair": 17.0, "dipole": 16.0, "liquid": 72.0}[case["system"]]
    if case["system"] == "liquid":
        inside = 4.0 / 3.0 * math.pi * 0.0218 * 7.0 ** 3 if N >= 1000 else math.pi / 6.0 * N
        pairs = 0.5 * N * inside
    exch = 19.0 * N2 if case.get("bosonic", True) else 0.0
    state = 8.0 * D * N * P * R
    if case["kind"] == "exchange":
        return {"bytes": 8.0 * D * 4 * N + 16.0 * D * N, "flops": 2.0 * exch}
    if case["kind"] == "observables":
        return {"bytes": 2 * state, "flops": P * pairs * (per + 20.0) + 2.0 * exch}
    return {"bytes": 5 * state, "flops": steps * R * (P * (pairs * per + 60.0 * D * N) + exch)}


# ------------------------------------------------- the same in plain 64 bits

RM, AZ_A, EPS, ALPHA, AZ_D, C6, C8, C10 = 5.60738, 0.5448504e6, 3.42016e-5, 13.353384, 1.241314, 1.3732412, 0.4253785, 0.1781


class _Exact:
    """R systems of one bead count, particles padded to the largest N
    (`on`: which are real): arrays [R][P][N][D]."""

    def __init__(self, systems):
        self.c = [s[0] for s in systems]
        c = self.c[0]
        R, P, D = len(systems), c["nbeads"], c["ndim"]
        self.R, self.P, self.D = R, P, D
        self.n = torch.tensor([q["natoms"] for q in self.c], device=DEV)
        N = self.N = int(self.n.max())
        self.on = torch.arange(N, device=DEV)[None] < self.n[:, None]
        self.x, self.p, self.f, self.fphys = (torch.zeros(R, P, N, D, dtype=F64, device=DEV) for _ in range(4))
        for r, (q, x, p) in enumerate(systems):
            self.x[r, :, :q["natoms"]], self.p[r, :, :q["natoms"]] = x, p
        self.fx = torch.zeros(R, 2, N, D, dtype=F64, device=DEV)
        self.beta = torch.tensor([1.0 / q["temperature"] for q in self.c], dtype=F64, device=DEV)
        self.bex = self.beta / P
        self.mass, self.dt, self.L = c["mass"], c["dt"], c["size"]
        self.omega = P / self.beta
        self.kappa = self.mass * self.omega ** 2
        self.pbc, self.bosonic = bool(c["pbc"]), bool(c["bosonic"]) and P > 1
        gamma = 1.0 / (100.0 * self.dt)
        self.c1 = math.exp(-0.5 * gamma * self.dt)
        self.c2 = torch.sqrt((1 - self.c1 ** 2) * self.mass / self.bex)
        self.cut = c["cutoff"] if not self.pbc or c["cutoff"] < 0 else min(c["cutoff"], 0.5 * self.L)
        if c["propagator"] == "normal_modes" or c["nmthermostat"]:
            k, b = torch.arange(P, dtype=F64, device=DEV)[:, None], torch.arange(P, dtype=F64, device=DEV)[None]
            kb = 2 * math.pi * torch.remainder(k * b, P) / P
            m = math.sqrt(2.0 / P) * torch.where(k < 0.5 * P, torch.cos(kb), -torch.sin(kb))
            m[0] = 1 / math.sqrt(P)
            if P % 2 == 0:
                m[P // 2] = (1 - 2 * torch.remainder(b[0], 2)) / math.sqrt(P)
            self.modes = m
        if c["thermostat"].startswith("nose"):
            chains = (R, P, N, D) if c["thermostat"].endswith("dim") else (R, P, N, 1)
            zeros = [[torch.zeros(chains, dtype=F64, device=DEV) for _ in range(c["nchains"])] for _ in range(3)]
            self.eta, self.etad, self.etadd = zeros

    def image(self, d):
        return d - self.L * torch.floor(d / self.L + 0.5) if self.pbc else d

    def col(self, v, dims):
        return v.reshape(-1, *([1] * dims))

    # external and pair forces, and with `energy` their energies and virials
    def physical(self, energy=False):
        c = self.c[0]
        kext = self.mass * c["ext_params"][0] ** 2 if c["ext_kind"] == "harmonic" else 0.0
        f = -kext * self.x
        v = 0.5 * kext * (self.x ** 2).sum((2, 3))
        w = kext * (self.x ** 2).sum((2, 3))
        vp, wp = torch.zeros_like(v), torch.zeros_like(v)
        kind = c["int_kind"]
        if kind == "harmonic":
            k = self.mass * c["int_params"][0] ** 2
            f = f - k * (self.x * self.col(self.n, 3) - self.x.sum(2, keepdim=True))
        elif kind != "free":
            N = self.N
            rows = max(1, min(N, (1 << 24) // N))
            for b in range(self.P):
                x = self.x[0, b]
                for i0 in range(0, N, rows):
                    xi = x[i0:i0 + rows]
                    d = self.image(xi[:, None] - x[None])
                    r2 = (d * d).sum(2)
                    i = torch.arange(i0, i0 + len(xi), device=DEV)
                    self_pair = i[:, None] == torch.arange(N, device=DEV)[None]
                    r2[self_pair] = 1.0
                    r = torch.sqrt(r2)
                    if kind == "dipole":
                        val = c["int_params"][0] / (r2 * r)
                        s = -3.0 * val / r2
                    else:
                        rs = r / RM
                        i2 = 1.0 / (rs * rs)
                        i6 = i2 ** 3
                        t = AZ_D / rs - 1.0
                        F = torch.where(rs < AZ_D, torch.exp(-t * t), torch.ones_like(t))
                        dF = torch.where(rs < AZ_D, 2 * AZ_D * i2 * t * F, torch.zeros_like(t))
                        rep = AZ_A * torch.exp(-ALPHA * rs)
                        att = i6 * (C6 + i2 * (C8 + i2 * C10))
                        tail = i6 / rs * (6 * C6 + i2 * (8 * C8 + i2 * 10 * C10))
                        s = EPS / RM * (-ALPHA * rep + tail * F - att * dF) / r
                        val = EPS * (rep - att * F)
                    drop = self_pair if self.cut < 0 else self_pair | ~(r < self.cut)
                    s = s.masked_fill(drop, 0.0)
                    f[0, b, i0:i0 + rows] -= (s[:, :, None] * d).sum(1)
                    if energy:
                        late = torch.arange(N, device=DEV)[None] > i[:, None]  # each pair once, seen from its first
                        vp[0, b] += val.masked_fill(drop | ~late, 0.0).sum()
                        wp[0, b] += (xi * ((s * late)[:, :, None] * d).sum(1)).sum()
        if energy:
            return f, v, w, vp, wp
        return f

    def exchange(self):
        """V_B, the exterior spring forces of beads 1 and P, and what the estimators need."""
        R, N, n, bex = self.R, self.N, self.n, self.bex
        x1, xP = self.x[:, 0], self.x[:, -1]
        link = (self.image(x1[:, 1:] - xP[:, :-1]) ** 2).sum(2)
        d = self.image(xP[:, :, None] - x1[:, None])  # [R][v][u]
        c2 = (d * d).sum(3)
        E = torch.zeros(R, N, N, dtype=F64, device=DEV)
        lead = torch.cat([torch.zeros(R, 1, dtype=F64, device=DEV), torch.cumsum(link, 1)], 1)
        E = 0.5 * self.col(self.kappa, 2) * ((lead[:, :, None] - lead[:, None]) + c2)
        V = torch.zeros(R, N + 1, dtype=F64, device=DEV)
        be = self.col(bex, 1)
        for m in range(1, N + 1):
            V[:, m] = -(torch.logsumexp(-be * (E[:, m - 1, :m] + V[:, :m]), 1) - math.log(m)) / bex
        Vb = torch.zeros(R, N + 1, dtype=F64, device=DEV)
        logq = torch.log(torch.arange(1, N + 1, dtype=F64, device=DEV))
        ninf = torch.tensor(-math.inf, dtype=F64, device=DEV)
        for l in range(N - 1, 0, -1):
            t = -be * (E[:, l:, l] + Vb[:, l + 1:]) - logq[None, l:]
            t = torch.where(self.on[:, l:], t, ninf)
            v = -torch.logsumexp(t, 1) / bex
            Vb[:, l] = torch.where(l < n, v, torch.zeros_like(v))
        VN = V.gather(1, n[:, None])
        be2 = self.col(bex, 2)
        real = self.on[:, :, None] & self.on[:, None]
        Pr = torch.exp(-be2 * (V[:, None, :N] + E + Vb[:, 1:, None] - VN[:, :, None]) - logq[None, :, None])
        low = torch.tril(torch.ones(N, N, dtype=torch.bool, device=DEV))
        Pr = torch.where(low[None] & real, Pr, torch.zeros_like(Pr))
        cut = 1.0 - torch.exp(-be * (V[:, 1:] + Vb[:, 1:] - VN))
        k = torch.arange(N - 1, device=DEV)
        Pr[:, k, k + 1] = torch.where(real[:, k, k + 1], cut[:, :-1], torch.zeros_like(cut[:, :-1]))
        pull = torch.zeros(R, 2, N, self.D, dtype=F64, device=DEV)
        for a in range(self.D):
            pull[:, 1, :, a] = -(Pr * d[..., a]).sum(2)
            pull[:, 0, :, a] = (Pr * d[..., a]).sum(1)
        pull[:, 0] += self.image(self.x[:, 1 % self.P] - x1)
        pull[:, 1] += self.image(self.x[:, self.P - 2] - xP)
        self.fx = self.col(self.kappa, 3) * pull
        return E, V, VN[:, 0]

    def estimators(self, E, V, VN):
        G = torch.zeros_like(V)
        be = self.col(self.bex, 1)
        for m in range(1, self.N + 1):
            w = torch.exp(-be * (E[:, m - 1, :m] + V[:, :m] - V[:, m:m + 1])) / m
            G[:, m] = ((G[:, :m] - E[:, m - 1, :m]) * w).sum(1)
        E0 = E[0]
        dist = math.exp(-float(self.bex[0] * (torch.diagonal(E0).sum() - VN[0])) - math.lgamma(self.N + 1))
        longest = math.exp(-float(self.bex[0] * (E0[self.N - 1, 0] - VN[0])))
        return float(G[0, self.N]) / self.P, dist, longest

    def perm_exchange(self):
        """The sum over permutations, by subsets of the first links' targets."""
        N = self.N
        d = self.image(self.x[0, 0][None] - self.x[0, -1][:, None])  # [l][m]: x1_m - xP_l
        d2 = (d * d).sum(2).cpu().numpy()
        e = 0.5 * float(self.kappa[0]) * float(self.bex[0]) * d2
        size = 1 << N
        fwd, bwd = np.full(size, -np.inf), np.full(size, -np.inf)
        fwd[0], bwd[size - 1] = 0.0, 0.0
        count = np.array([bin(m).count("1") for m in range(size)])
        bits = np.arange(N)
        masks = np.arange(size)
        for l in range(N):
            for m in bits:
                src = masks[(count == l) & ((masks >> m) & 1 == 0)]
                fwd[src | (1 << m)] = np.logaddexp(fwd[src | (1 << m)], fwd[src] - e[l, m])
        for l in range(N - 1, -1, -1):
            for m in bits:
                src = masks[(count == l) & ((masks >> m) & 1 == 0)]
                bwd[src] = np.logaddexp(bwd[src], bwd[src | (1 << m)] - e[l, m])
        M = np.zeros((N, N))
        for l in range(N):
            for m in bits:
                src = masks[(count == l) & ((masks >> m) & 1 == 0)]
                M[l, m] = np.exp(fwd[src] + bwd[src | (1 << m)] - e[l, m] - fwd[size - 1]).sum()
        M = torch.tensor(M, dtype=F64, device=DEV)
        fP = (M[:, :, None] * d).sum(1) + self.image(self.x[0, self.P - 2] - self.x[0, -1])
        f1 = -(M[:, :, None] * d).sum(0) + self.image(self.x[0, 1 % self.P] - self.x[0, 0])
        self.fx = self.kappa[0] * torch.stack([f1, fP])[None]

    def forces(self):
        self.fphys = self.physical()
        x = self.x
        spring = self.image(torch.roll(x, 1, 1) - x) + self.image(torch.roll(x, -1, 1) - x)
        spring = self.col(self.kappa, 3) * spring
        if self.bosonic:
            self.perm_exchange() if self.c[0]["exchange"] == "factorial" else self.exchange()
            spring[:, 0], spring[:, -1] = self.fx[:, 0], self.fx[:, 1]
        self.f = (spring + self.fphys) * self.on[:, None, :, None]

    # Philox4x32-10 and Box-Muller in correctly rounded 32-bit arithmetic: the
    # library's normals are these by definition
    def normals(self, t):
        f = lambda v: torch.tensor(v, dtype=torch.float32, device=DEV)  # noqa: E731
        fma = lambda a, b, c: (a.double() * b.double() + c.double()).float()  # noqa: E731
        half = (self.n + 1) // 2
        H = int(half.max())
        # pair index (bead D + axis) ceil(N / 2) + pair, by replica
        line = torch.arange(self.P * self.D, device=DEV).reshape(1, -1, 1)
        k = line * half[:, None, None] + torch.arange(H, device=DEV)
        rep = torch.tensor([c["replica"] for c in self.c], device=DEV)[:, None, None].expand_as(k)
        w = [k, rep, torch.full_like(k, t & 0xffffffff), torch.full_like(k, t >> 32)]
        seed = self.c[0]["seed"]
        k0, k1 = seed & 0xffffffff, seed >> 32

        def mul(m, v):
            lo, hi = m * (v & 0xffff), m * (v >> 16)
            mid = hi + (lo >> 16)
            return mid >> 16, ((mid & 0xffff) << 16) | (lo & 0xffff)

        for _ in range(10):
            h0, l0 = mul(0xD2511F53, w[0])
            h1, l1 = mul(0xCD9E8D57, w[2])
            w = [h1 ^ w[1] ^ k0, l1, h0 ^ w[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
        u = ((w[0] >> 8) + 1).float() * f(2.0 ** -24)
        man, ex = torch.frexp(u)
        man, ex = man * 2, ex - 1
        big = man > f(1.41421354)
        man, ex = torch.where(big, man * f(0.5), man), torch.where(big, ex + 1, ex)
        sv = (man - 1) / (man + 1)
        s2 = sv * sv
        q = f(0.111111112).expand_as(s2)
        for a in (0.142857149, 0.2, 0.333333343, 1.0):
            q = fma(q, s2, f(a))
        ef = ex.float()
        ln = fma(ef, f(0.693145752), fma(ef, f(1.42860677e-06), (2 * sv) * q))
        rad = torch.sqrt((f(-2.0) * ln).double()).float()
        quad, ph = w[2] >> 30, (((w[2] >> 6) & 0xffffff).float() * f(2.0 ** -24)) * f(1.57079637)
        p2 = ph * ph
        sp, cp = f(1.60590444e-10).expand_as(p2), f(-1.14707454e-11).expand_as(p2)
        for a in (-2.50521079e-08, 2.75573188e-06, -1.98412701e-04, 8.33333377e-03, -0.166666672):
            sp = fma(sp, p2, f(a))
        sp = fma(sp * p2, ph, ph)
        for a in (2.08767559e-09, -2.75573188e-07, 2.48015876e-05, -1.38888892e-03, 4.16666679e-02, -0.5, 1.0):
            cp = fma(cp, p2, f(a))
        odd = (quad & 1) == 1
        sn, cs = torch.where(odd, cp, sp), torch.where(odd, sp, cp)
        sn, cs = torch.where((quad & 2) != 0, -sn, sn), torch.where(((quad + 1) & 2) != 0, -cs, cs)
        z = torch.stack([rad * cs, rad * sn], 3).double().reshape(self.R, self.P, self.D, 2 * H)
        z = torch.nn.functional.pad(z, (0, max(0, self.N - 2 * H)))[..., :self.N]
        return z.transpose(2, 3)

    def to_modes(self, v):
        return torch.einsum("kb,rbnd->rknd", self.modes, v)

    def from_modes(self, v):
        return torch.einsum("kb,rknd->rbnd", self.modes, v)

    def thermostat(self, t):
        c = self.c[0]
        if c["thermostat"] == "langevin":
            p = self.to_modes(self.p) if c["nmthermostat"] else self.p
            p = self.c1 * p + self.col(self.c2, 3) * self.normals(t)
            self.p = self.from_modes(p) if c["nmthermostat"] else p
        elif c["thermostat"] != "none":
            self.chains()
        self.p = self.p * self.on[:, None, :, None]
        com = self.p.sum((1, 2)) / (self.n * self.P)[:, None].to(F64)
        self.p = (self.p - com[:, None, None]) * self.on[:, None, :, None]

    def chains(self):
        """One step of the Nose-Hoover chains (Tuckerman et al., J. Phys. A 39, 5629, 2006)."""
        kt, dt = float(1.0 / self.bex[0]), self.dt
        Q = float(self.beta[0]) / self.P
        per = 1 if self.eta[0].shape[3] == self.D else self.D
        e2 = (self.p ** 2 if per == 1 else (self.p ** 2).sum(3, keepdim=True)) / self.mass
        need, Q1, M = per * kt, per * Q, len(self.eta)
        eta, v, a = self.eta, self.etad, self.etadd
        a[0] = (e2 - need) / Q1
        v[M - 1] = v[M - 1] + a[M - 1] * 0.25 * dt
        for i in range(M - 2, -1, -1):
            g = torch.exp(-0.125 * dt * v[i + 1])
            v[i] = (v[i] * g + a[i] * 0.25 * dt) * g
        s = torch.exp(-0.5 * dt * v[0])
        for i in range(M):
            eta[i] = eta[i] + 0.5 * dt * v[i]
        a[0] = (e2 * s * s - need) / Q1
        v[0] = (v[0] * g + a[0] * 0.25 * dt) * g
        former = Q1
        for i in range(1, M - 1):
            g = torch.exp(-0.125 * dt * v[i + 1])
            v[i] = v[i] * g
            a[i] = (former * v[i - 1] ** 2 - kt) / Q
            v[i] = (v[i] + a[i] * 0.25 * dt) * g
            former = Q
        a[M - 1] = (Q * v[M - 2] ** 2 - kt) / Q
        v[M - 1] = v[M - 1] + a[M - 1] * 0.25 * dt
        self.p = self.p * s

    def kick(self):
        """The half-kick of the normal-mode propagator."""
        f = self.fphys.clone()
        if self.bosonic:
            x, k = self.x, self.col(self.kappa, 2)
            for side, b in ((0, 0), (1, self.P - 1)):
                inner = -k * (2 * x[:, b] - x[:, b - 1] - x[:, (b + 1) % self.P])
                f[:, b] += self.fx[:, side] - inner
        self.p = self.p + 0.5 * self.dt * f

    def step(self, t):
        self.thermostat(2 * t)
        if self.c[0]["propagator"] == "normal_modes":
            self.kick()
            q, p = self.to_modes(self.x), self.to_modes(self.p)
            w = 2 * self.omega[:, None] * torch.sin(torch.arange(self.P, dtype=F64, device=DEV) * math.pi / self.P)[None]
            w = w[:, :, None, None]
            c, s = torch.cos(w * self.dt), torch.sin(w * self.dt)
            free = w == 0
            drift = torch.where(free, torch.full_like(w, self.dt / self.mass), s / (self.mass * (w + free)))
            q, p = c * q + drift * p, -self.mass * w * s * q + c * p
            self.x, self.p = self.from_modes(q), self.from_modes(p)
            self.forces()
            self.kick()
        else:
            self.p = self.p + 0.5 * self.dt * self.f
            self.x = self.x + self.dt * self.p / self.mass
            self.forces()
            self.p = self.p + 0.5 * self.dt * self.f
        self.thermostat(2 * t + 1)


def _exact_observables(e):
    f, v, w, vp, wp = e.physical(energy=True)
    P, N, D, x = e.P, e.N, e.D, e.x
    beta, kappa = float(e.beta[0]), float(e.kappa[0])
    spring = 0.5 * kappa * (e.image(torch.roll(x, 1, 1) - x) ** 2).sum((2, 3))[0]
    ke = (e.p ** 2).sum() / (2 * e.mass)
    E, V, VN = e.exchange()
    prim, dist, longest = e.estimators(E, V, VN)
    even = torch.arange(P, device=DEV) % 2 == 0
    pot = (v + vp)[0]
    f2 = (f ** 2).sum((2, 3))[0]
    gsf = torch.where(even, pot / (3 * P) + f2 / (9 * kappa * P), -pot / (3 * P)).sum() * -beta
    val = dict(kinetic=0.5 * D * N / beta * P + prim - spring[1:].sum() / P, potential=pot.sum() / P,
               ext_pot=v.sum() / P, int_pot=vp.sum() / P, virial=0.5 * (w + wp).sum() / P,
               temperature=2 * ke / (D * N * P) / P / KELVIN, cl_kinetic=ke, cl_spring=spring[1:].sum() + VN[0],
               prob_dist=dist, prob_all=longest, w_gsf=gsf, pot_gsf=pot[~even].sum() / (0.5 * P), nh_energy=0.0)
    return {k: np.float64(float(q)) for k, q in val.items()}


def exact(case, seed):
    systems = _inputs(case, seed)
    if case["kind"] == "ensemble":
        done = {}
        for P in sorted({s[0]["nbeads"] for s in systems}):
            at = [r for r, s in enumerate(systems) if s[0]["nbeads"] == P]
            e = _Exact([systems[r] for r in at])
            for t in range(case["steps"]):
                e.step(t)
            for k, r in enumerate(at):
                n = systems[r][0]["natoms"]
                done[r] = [v[k, :, :n].cpu().numpy().ravel() for v in (e.x, e.p, e.f)]
        return [np.concatenate([done[r][k] for r in range(len(systems))]) for k in range(3)]
    e = _Exact(systems)
    if case["kind"] == "observables":
        return _exact_observables(e)
    if case["kind"] == "exchange":
        E, V, VN = e.exchange()
        prim, dist, longest = e.estimators(E, V, VN)
        return dict(VB=np.float64(float(VN[0])), prim=np.float64(prim), p_distinct=np.float64(dist),
                    p_longest=np.float64(longest), f1=e.fx[0, 0].cpu().numpy(), fP=e.fx[0, 1].cpu().numpy())
    for t in range(case["steps"]):
        e.step(t)
    return [v[0] for v in (e.x, e.p, e.f)]
