"""Timed workloads of the engine: what its users have it do, through its public entry points.

A case is a dict of plain values. `kind` says which entry point it times:

  rhs       Engine.accel, the drop-in right-hand side that a host integrator calls once per stage
  run       Engine.run: upload a state, advance it, download frames and the final state
  energy    Engine.energy: the energies and temperature of one saved frame
  rdf       rdf_histogram over the saved frames of a trajectory
  gradient  Engine.ml_batch_gradient: loss and gradient of the learned model on one training batch

`system` is one of

  lj       Lennard-Jones liquid at density 0.8 in a cubic box (reduced units, cutoff 2.5)
  water    SPC/Fw water at 300 K in a cubic box (kJ/mol, nm, ps)
  gravity  Plummer sphere (G = M = 1), equal or uneven masses
  ions     unbounded charged particles with the untruncated Coulomb force, optionally with a
           Lennard-Jones term
  batch    replicas of the Lennard-Jones liquid of uneven sizes and temperatures, Langevin (BAOAB)

exact() restates each of them in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

import __graft_entry__

nbg = __graft_entry__.load_package()

WATER = dict(rOH=0.1012, aHOH=113.24 * math.pi / 180, eps=0.650299, sigma=0.3165492, R=0.9, qO=-0.82, qH=0.41)
ND, NH = 64, 128  # inputs and hidden width of the learned model


def listed():
    return [
        # a host integrator's right-hand side on the standard small liquid, from page-locked buffers
        dict(name="rhs_lj_1000", kind="rhs", system="lj", n=1000, pinned=True, thermostat="none"),
        # free ions in open space: every pair interacts, host buffers as an adaptive solver holds them
        dict(name="rhs_ions_5000", kind="rhs", system="ions", n=5000, pinned=False, lj=False, thermostat="none"),
        # the standard small liquid run at constant energy, some frames kept
        dict(name="run_lj_1000", kind="run", system="lj", n=1000, steps=200, save_every=20, thermostat="none"),
        # an ordinary liquid under a thermostat, frames kept for analysis
        dict(name="run_lj_10976_nosehoover", kind="run", system="lj", n=10976, steps=200, save_every=20,
             thermostat="nosehoover"),
        # a small water box: fewer than three cutoffs across, so every pair is tested
        dict(name="run_water_216", kind="run", system="water", n_mol=216, steps=100, save_every=20,
             thermostat="berendsen"),
        # the water benchmark's box
        dict(name="run_water_4096", kind="run", system="water", n_mol=4096, steps=100, save_every=0,
             thermostat="berendsen"),
        # a star cluster with a mass spectrum
        dict(name="run_gravity_1500", kind="run", system="gravity", n=1500, steps=200, save_every=20,
             equal_mass=False, thermostat="none"),
        # the headline benchmark's sphere
        dict(name="run_gravity_65536", kind="run", system="gravity", n=65536, steps=8, save_every=0,
             equal_mass=True, thermostat="none"),
        # the replica ensemble of the benchmark
        dict(name="run_batch_256", kind="run", system="batch", replicas=256, n_min=256, n_max=8192, steps=20,
             save_every=0, thermostat="langevin"),
        # energy conservation check of one frame of a water run
        dict(name="energy_water_4096", kind="energy", system="water", n_mol=4096, thermostat="berendsen"),
        # oxygen-oxygen radial distribution over the frames of a water run
        dict(name="rdf_water_4096x64", kind="rdf", n_mol=4096, frames=64, maxbin=1000),
        # one training batch of the learned short-range model
        dict(name="gradient_2048", kind="gradient", species=1, batch=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "run", "run", "run", "run", "energy", "energy", "rdf", "gradient"])
    if kind == "rdf":
        n_mol = _log(rng, 100, 6000)
        return dict(kind=kind, n_mol=n_mol, frames=max(1, min(400, int(rng.uniform(0.1, 1.0) * 1.0e9 / n_mol ** 2))),
                    maxbin=rng.randint(50, 1500))
    if kind == "gradient":
        return dict(kind=kind, species=rng.randint(0, 1), batch=_log(rng, 100, 16384))
    if kind == "energy":
        system = rng.choice(["lj", "water", "gravity", "ions"])
    elif kind == "rhs":
        system = rng.choice(["lj", "water", "gravity", "ions", "ions"])
    else:
        system = rng.choice(["lj", "lj", "water", "water", "gravity", "batch"])
    case = dict(kind=kind, system=system)
    if system == "lj":
        case["n"] = _log(rng, 108, 100000)
        case["thermostat"] = rng.choice(["none", "berendsen", "nosehoover", "andersen"])
        size = case["n"] if case["n"] > 480 else 80 * case["n"]  # below: a box of fewer than three cutoffs
    elif system == "water":
        case["n_mol"] = _log(rng, 216, 12000)
        case["thermostat"] = rng.choice(["none", "berendsen", "nosehoover"])
        size = 10 * case["n_mol"] if case["n_mol"] > 900 else 220 * case["n_mol"]
    elif system == "gravity":
        case["n"] = _log(rng, 50, 8192 if kind == "energy" else 40000)
        case["equal_mass"] = rng.random() < 0.5
        case["thermostat"] = "none"
        size = case["n"] ** 2 / 3000
    elif system == "ions":
        case["n"] = _log(rng, 50, 8192 if kind == "energy" else 12000)
        case["lj"] = rng.random() < 0.3
        case["thermostat"] = "none"
        size = case["n"]
    else:
        case["replicas"] = _log(rng, 4, 128)
        case["n_min"] = rng.randint(128, 512)
        case["n_max"] = _log(rng, 600, 8192)
        case["thermostat"] = "langevin"
        size = 200000
    if kind == "rhs":
        case["pinned"] = rng.random() < 0.5
    if kind == "run":
        case["steps"] = max(4, min(rng.randint(10 if system == "batch" else 40, 300), int(4.0e6 / size)))
        case["save_every"] = rng.choice([0, 5, 10, 20]) if size < 20000 and system != "batch" else 0
    return case


# ------------------------------------------------------------------ inputs

def _masses(case, n, seed):
    m = np.ones(n)
    if not case.get("equal_mass", True):
        m = np.random.default_rng(seed + 77).uniform(0.2, 1.8, n)
    return m


def _thermostat(case, T):
    return {"none": nbg.NullThermostat(), "berendsen": nbg.BerendsenThermostat(T, 0.1),
            "nosehoover": nbg.NoseHooverThermostat(T, 0.5), "andersen": nbg.AndersenThermostat(T, 2.0)}[case["thermostat"]]


def _inputs(case, seed):
    """Positions, velocities and the numbers that describe the system."""
    system = case["system"]
    w = nbg.workloads
    if system == "lj":
        u, v, L = w.lj_argon_lattice(case["n"], rho=0.8, T=1.0, seed=seed, jitter=0.05)
        return dict(u=u, v=v, L=L, m=np.ones(case["n"]), dt=0.004, kb=1.0, T0=0.9)
    if system == "water":
        u, v, L = w.spcfw_water_box(case["n_mol"], seed=seed, T=300.0)
        n = case["n_mol"]
        # vibrating molecules: the box's own start from their equilibrium geometry
        u = u + np.random.default_rng(seed + 9).standard_normal(u.shape) * np.tile([0.001, 0.003, 0.003], n)[:, None]
        return dict(u=u, v=v, L=L, m=np.tile([w.M_O, w.M_H, w.M_H], n), dt=0.0005, kb=w.KB_KJ, T0=300.0,
                    q=np.tile([WATER["qO"], WATER["qH"], WATER["qH"]], n))
    if system == "gravity":
        u, v, m = w.plummer_sphere(case["n"], seed=seed)
        if not case["equal_mass"]:
            m = m * _masses(case, case["n"], seed)
        return dict(u=u, v=v, L=0.0, m=m, dt=1e-3, kb=1.0)
    if system == "ions":
        n = case["n"]
        u, v, L = w.lj_argon_lattice(n, rho=0.3, T=1.0, seed=seed, jitter=0.1)
        q = np.where(np.random.default_rng(seed + 5).permutation(n) % 2 == 0, 1.0, -1.0)
        return dict(u=u - 0.5 * L, v=v, L=0.0, m=np.ones(n), dt=0.001, kb=1.0, q=q, k=1.5)
    raise ValueError(system)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()


def _engine(case, s):
    """The handle that a program keeps for its system."""
    system = case["system"]
    if system == "lj":
        desc, keep = nbg.lennard_jones_descriptor(s["m"], s["L"], thermostat=_thermostat(case, s["T0"]), seed=11)
        return nbg.Engine(desc), keep
    u, v, m = s["u"], s["v"], s["m"]
    if system == "water":
        sysm = nbg.WaterSPCFw(nbg.workloads.water_molecules(u, v), nbg.workloads.M_H, nbg.workloads.M_O, WATER["qH"],
                              WATER["qO"], nbg.LennardJonesParameters(WATER["eps"], WATER["sigma"], WATER["R"]),
                              nbg.ElectrostaticParameters(nbg.workloads.K_EL, WATER["R"]),
                              nbg.SPCFwParameters(WATER["rOH"], WATER["aHOH"], nbg.workloads.SPCFW_KB,
                                                  nbg.workloads.SPCFW_KA))
        sim = nbg.NBodySimulation(sysm, (0.0, 1.0), nbg.CubicPeriodicBoundaryConditions(s["L"]),
                                  _thermostat(case, s["T0"]), kb=s["kb"], skin=0.1, rebuild_every=0)
    elif system == "gravity":
        bodies = [nbg.MassBody(u[i], v[i], m[i]) for i in range(len(m))]
        sim = nbg.NBodySimulation(nbg.GravitationalSystem(bodies, 1.0), (0.0, 1.0), kb=s["kb"])
    else:
        bodies = [nbg.ChargedParticle(u[i], v[i], m[i], s["q"][i]) for i in range(len(m))]
        if case["lj"]:
            sysm = nbg.PotentialNBodySystem(bodies, {"lennard_jones": nbg.LennardJonesParameters(1.0, 1.0, 2.5),
                                                     "electrostatic": nbg.ElectrostaticParameters(s["k"])})
        else:
            sysm = nbg.ChargedParticles(bodies, s["k"])
        sim = nbg.NBodySimulation(sysm, (0.0, 1.0), kb=s["kb"])
    desc, keep = nbg.system_descriptor(sim)
    return nbg.Engine(desc), keep


def _batch(case, seed):
    """Replicas of uneven sizes (the case's) and temperatures, one of them of the largest size."""
    rng = np.random.default_rng(case["replicas"])
    sizes = rng.integers(case["n_min"], case["n_max"] + 1, size=case["replicas"])
    sizes[rng.integers(case["replicas"])] = case["n_max"]
    rng = np.random.default_rng(seed)
    out = []
    for r, n in enumerate(sizes):
        T = float(rng.uniform(0.7, 1.5))
        pos, vel, L = nbg.workloads.lj_argon_lattice(int(n), rho=0.8, T=T, seed=seed * 100003 + r, jitter=0.02)
        out.append(dict(pos=pos, vel=vel, L=L, T=T, n=int(n)))
    return out


def _frames(case, seed):
    """Frames of a water trajectory: one box, its molecules displaced afresh in every frame."""
    u, _, L = nbg.workloads.spcfw_water_box(case["n_mol"], seed=seed, T=300.0)
    rng = np.random.default_rng(seed + 3)
    shift = rng.standard_normal((case["frames"], case["n_mol"], 1, 3)) * 0.08
    return (u.reshape(1, -1, 3, 3) + shift).reshape(case["frames"], -1, 3), L


def _gradient_inputs(case, seed):
    rng = np.random.default_rng(seed)
    B = case["batch"]
    theta = np.concatenate([rng.standard_normal(ND * NH) / 8, 0.1 * rng.standard_normal(NH),
                            rng.standard_normal(NH * NH) / math.sqrt(NH), 0.1 * rng.standard_normal(NH),
                            rng.standard_normal(NH) / math.sqrt(NH), np.zeros(1),
                            np.zeros(ND), np.ones(ND), np.zeros(1), np.ones(1)]).astype(np.float32)
    return (theta, rng.standard_normal((B, ND)).astype(np.float32), rng.standard_normal(B).astype(np.float32))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "rdf":
        frames, L = _frames(case, seed)
        return dict(case=case, frames=frames, L=L, idx=np.arange(0, 3 * case["n_mol"], 3))
    if kind == "gradient":
        theta, x, y = _gradient_inputs(case, seed)
        water = dict(system="water", n_mol=1000, thermostat="none")
        engine, keep = _engine(water, _inputs(water, 1))
        engine.ml_enable()
        engine.ml_set_params(case["species"], theta)
        return dict(case=case, engine=engine, keep=keep, x=x, y=y)
    if case["system"] == "batch":
        reps = _batch(case, seed)
        descs, keep = [], []
        for r, rep in enumerate(reps):
            d, k = nbg.lennard_jones_descriptor(np.ones(rep["n"]), rep["L"], skin=0.5, seed=1000 + r,
                                                thermostat=nbg.LangevinThermostat(rep["T"], 1.0))
            d.flags |= nbg._abi.NBG_FLAG_LANGEVIN_BAOAB
            descs.append(d)
            keep.append(k)
        return dict(case=case, engine=nbg.Engine(descs), keep=keep, u=np.concatenate([r["pos"] for r in reps]),
                    v=np.concatenate([r["vel"] for r in reps]), dt=0.005)
    s = _inputs(case, seed)
    s["engine"], s["keep"] = _engine(case, s)
    if case["thermostat"] == "nosehoover":  # the thermostat's own column
        s["u"] = np.concatenate([s["u"], np.zeros((1, 3))])
        s["v"] = np.concatenate([s["v"], np.zeros((1, 3))])
    s["case"] = case
    if kind == "rhs":
        s["dv"] = np.zeros_like(s["u"])
        if case["pinned"]:
            for k in ("u", "v", "dv"):
                s[k] = _pinned(s[k])
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhs":
        return state["engine"].accel(state["v"], state["u"], out=state["dv"])
    if kind == "run":
        u, v, tu, tv, _ = state["engine"].run(state["u"], state["v"], state["dt"], case["steps"], case["save_every"],
                                              save_trajectory=case["save_every"] > 0, step=0)
        return {"u": u, "v": v, "frames_u": tu, "frames_v": tv} if tu is not None else {"u": u, "v": v}
    if kind == "energy":
        return state["engine"].energy(state["u"], state["v"])
    if kind == "rdf":
        return nbg._abi.rdf_histogram(state["frames"], state["idx"], state["L"], case["maxbin"])
    loss, grad = state["engine"].ml_batch_gradient(case["species"], state["x"], state["y"])
    return {"loss": loss, "grad": grad}


# ------------------------------------------------------------------ work

def _pairs(case):
    """Unordered pairs whose interaction one evaluation of the forces (or energies) holds, and flops of each."""
    system = case["system"]
    if system == "lj":
        n = case["n"]
        inside = min(0.5 * n * (n - 1), 0.5 * n * 0.8 * 4.0 / 3.0 * math.pi * 2.5 ** 3)
        return n, 27.0 * inside
    if system == "water":
        n = 3 * case["n_mol"]
        inside = min(0.5 * n * (n - 3), 0.5 * n * 100.0 * 4.0 / 3.0 * math.pi * WATER["R"] ** 3)
        return n, 23.0 * inside + 120.0 * case["n_mol"]
    n = case["n"]
    return n, 23.0 * 0.5 * n * (n - 1)


def work(case):
    kind = case["kind"]
    if kind == "rdf":
        n = case["n_mol"]
        return {"bytes": 24.0 * n * case["frames"] + 8.0 * case["maxbin"], "flops": 16.0 * 0.5 * n * (n - 1) * case["frames"]}
    if kind == "gradient":
        B, p = case["batch"], ND * NH + 3 * NH + NH * NH + 1
        return {"bytes": 4.0 * (B * (ND + 1) + 2 * p), "flops": 2.0 * B * (2 * ND * NH + 3 * NH * NH + 4 * NH)}
    if case["system"] == "batch":
        n = case["replicas"] * 0.5 * (case["n_min"] + case["n_max"])
        pair = 27.0 * 0.5 * n * 0.8 * 4.0 / 3.0 * math.pi * 2.5 ** 3
        return {"bytes": 96.0 * n, "flops": (case["steps"] + 1) * (pair + 40.0 * n)}
    n, flops = _pairs(case)
    if kind == "rhs":
        return {"bytes": 48.0 * n, "flops": flops}
    if kind == "energy":
        return {"bytes": 48.0 * n, "flops": flops}
    frames = case["steps"] // case["save_every"] if case["save_every"] else 0
    return {"bytes": 96.0 * n + 48.0 * n * frames, "flops": (case["steps"] + 1) * (flops + 24.0 * n)}


# ------------------------------------------------------------------ the same in 64 bits

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEVICE)


class _Exact:
    """Forces and energies of one system by all pairs in 64 bits."""

    def __init__(self, case, s):
        self.case, self.system, self.L = case, case["system"], s["L"]
        self.m = _t(s["m"])
        self.n = len(self.m)
        self.q = _t(s["q"]) if "q" in s else None
        water = self.system == "water"
        self.k = nbg.workloads.K_EL if water else s.get("k", 0.0)
        self.eps, self.sig2, self.R = (WATER["eps"], WATER["sigma"] ** 2, WATER["R"]) if water else (1.0, 1.0, 2.5)
        self.has_lj = water or self.system == "lj" or bool(case.get("lj"))
        self.el_R = WATER["R"] if water else math.inf
        self.rows = max(1, min(self.n, int(2 ** 26 // self.n)))

    def _chunks(self, x):
        for a in range(0, self.n, self.rows):
            b = min(self.n, a + self.rows)
            d = x[a:b, None, :] - x[None, :, :]
            if self.L > 0:
                d = d - self.L * torch.round(d / self.L)
            r2 = (d * d).sum(-1)
            i = torch.arange(a, b, device=DEVICE)[:, None]
            j = torch.arange(self.n, device=DEVICE)[None, :]
            if self.system == "water":
                el, lj = i // 3 != j // 3, (i % 3 == 0) & (j % 3 == 0) & (i != j)
            else:
                el = lj = i != j
            r2 = torch.where(i == j, torch.ones_like(r2), r2)
            yield a, b, d, r2, el, lj

    def accel(self, x):
        f = torch.zeros_like(x)
        for a, b, d, r2, el, lj in self._chunks(x):
            zero = torch.zeros_like(r2)
            if self.system == "gravity":
                f[a:b] = -torch.einsum("ij,ijk->ik", torch.where(el, self.m[None, :] * r2 ** -1.5, zero), d)
                continue
            g = zero
            if self.has_lj:
                s6 = (self.sig2 / r2) ** 3
                g = g + torch.where(lj & (r2 < self.R ** 2), 24 * self.eps * (2 * s6 * s6 - s6) / r2, zero)
            if self.q is not None:
                g = g + torch.where(el & (r2 < self.el_R ** 2), self.k * self.q[a:b, None] * self.q[None, :] * r2 ** -1.5, zero)
            f[a:b] = torch.einsum("ij,ijk->ik", g, d)
        if self.system == "gravity":
            return f
        if self.system == "water":
            f = f + self._bonded(x)
        return f / self.m[:, None]

    def _bonded(self, x):
        w = x.view(-1, 3, 3)
        r1, r2 = w[:, 1] - w[:, 0], w[:, 2] - w[:, 0]
        n1, n2 = r1.norm(dim=1, keepdim=True), r2.norm(dim=1, keepdim=True)
        f1 = -nbg.workloads.SPCFW_KB * (n1 - WATER["rOH"]) * r1 / n1
        f2 = -nbg.workloads.SPCFW_KB * (n2 - WATER["rOH"]) * r2 / n2
        normal = torch.linalg.cross(r1, r2)
        p1, p2 = torch.linalg.cross(r1, normal), torch.linalg.cross(-r2, normal)
        t = -nbg.workloads.SPCFW_KA * (torch.arccos((r1 * r2).sum(1, keepdim=True) / (n1 * n2)) - WATER["aHOH"])
        f1 = f1 + p1 * t / (p1.norm(dim=1, keepdim=True) * n1)
        f2 = f2 + p2 * t / (p2.norm(dim=1, keepdim=True) * n2)
        return torch.stack([-f1 - f2, f1, f2], dim=1).reshape(-1, 3)

    def energies(self, x, v):
        lj_e = el_e = g_e = 0.0
        for a, b, d, r2, el, lj in self._chunks(x):
            zero = torch.zeros_like(r2)
            if self.system == "gravity":
                g_e -= 0.5 * float(torch.where(el, self.m[a:b, None] * self.m[None, :] / r2.sqrt(), zero).sum())
                continue
            if self.has_lj:
                s6 = (self.sig2 / r2.clamp(max=self.R ** 2)) ** 3
                lj_e += 2 * self.eps * float(torch.where(lj, s6 * s6 - s6, zero).sum())
            if self.q is not None:
                r = r2.sqrt().clamp(max=self.el_R)
                el_e += 0.5 * self.k * float(torch.where(el, self.q[a:b, None] * self.q[None, :] / r, zero).sum())
        bonds = angles = 0.0
        if self.system == "water":
            w = x.view(-1, 3, 3)
            r1, r2 = w[:, 1] - w[:, 0], w[:, 2] - w[:, 0]
            n1, n2 = r1.norm(dim=1), r2.norm(dim=1)
            bonds = 0.5 * nbg.workloads.SPCFW_KB * float(((n1 - WATER["rOH"]) ** 2 + (n2 - WATER["rOH"]) ** 2).sum())
            th = torch.arccos((r1 * r2).sum(1) / (n1 * n2))
            angles = 0.5 * nbg.workloads.SPCFW_KA * float(((th - WATER["aHOH"]) ** 2).sum())
        mv2 = float((self.m[:, None] * v * v).sum())
        potential = lj_e + el_e + bonds + angles
        return {"kinetic": 0.5 * mv2, "lennard_jones": lj_e, "electrostatic": el_e, "bonds": bonds, "angles": angles,
                "gravity": g_e, "potential": potential, "total": 0.5 * mv2 + potential}

    def ndf(self):
        return 3 * self.n - (2 * (self.n // 3) if self.system == "water" else 0)


def _philox(seed, atom, step, stream):
    """Philox4x32-10 of counter (atom, step, 0, stream) and key seed, on int64 tensors of 32-bit words."""
    m32 = 0xFFFFFFFF
    c = [atom & m32, torch.full_like(atom, step & m32), torch.full_like(atom, step >> 32), torch.full_like(atom, stream)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m32) ^ c[1] ^ k0, p1 & m32, ((p0 >> 32) & m32) ^ c[3] ^ k1, p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c


def _normals(seed, atom, step):
    a, b = _philox(seed, atom, step, 1), _philox(seed, atom, step, 2)
    s24 = 1.0 / 16777216.0
    u1, u2 = ((a[0] >> 8) + 1).double() * s24, (a[1] >> 8).double() * s24
    u3, u4 = ((b[0] >> 8) + 1).double() * s24, (b[1] >> 8).double() * s24
    r = torch.sqrt(-2 * torch.log(u1))
    return torch.stack([r * torch.cos(2 * math.pi * u2), r * torch.sin(2 * math.pi * u2),
                        torch.sqrt(-2 * torch.log(u3)) * torch.cos(2 * math.pi * u4)], dim=1)


def _exact_run(case, s):
    e, dt, therm = _Exact(case, s), s["dt"], case["thermostat"]
    x, v, n = _t(s["u"]), _t(s["v"]), len(s["m"])
    ndf, T0, kb = e.ndf(), s.get("T0"), s["kb"]
    nh = therm == "nosehoover"
    zeta = rate = 0.0

    def rhs(x, v):
        nonlocal rate
        a = e.accel(x)
        if therm in ("berendsen", "nosehoover"):
            T = float((e.m[:, None] * v * v).sum()) / (kb * ndf)
            if nh:
                a = a - zeta * v
                rate = (T / T0 - (ndf + 1.0) / ndf) / 0.5 ** 2
            else:
                a = a + 0.5 / 0.1 * (T0 / T - 1.0) * v
        return a

    def whole(t, z):
        t = t.cpu().numpy().copy()
        return np.concatenate([t, [[z, 0.0, 0.0]]]) if nh else t

    fu, fv = [whole(x, 0.0)], [whole(v, 0.0)]
    a = rhs(x, v)
    for k in range(case["steps"]):
        x = x + dt * v + dt * dt * (0.5 * a)
        zeta = zeta + dt * rate
        an = rhs(x, v)
        v = v + dt * (0.5 * a + 0.5 * an)
        a = an
        if therm == "andersen":
            atom = torch.arange(n, device=DEVICE)
            w = _philox(11, atom, k, 0)
            hit = ((w[0] >> 5).double() * 67108864.0 + (w[1] >> 6).double()) / 9007199254740992.0 < 2.0 * dt
            v = torch.where(hit[:, None], math.sqrt(kb * T0) * _normals(11, atom, k), v)
        if case["save_every"] and ((k + 1) % case["save_every"] == 0 or k + 1 == case["steps"]):
            fu.append(whole(x, zeta))
            fv.append(whole(v, rate))
    out = {"u": whole(x, zeta), "v": whole(v, rate)}
    if case["save_every"]:
        out["frames_u"], out["frames_v"] = np.stack(fu), np.stack(fv)
    return out


def _exact_batch(case, seed):
    dt, reps = 0.005, _batch(case, seed)
    c1 = math.exp(-dt)
    ends = np.cumsum([0] + [r["n"] for r in reps])
    forces = [_Exact(dict(system="lj"), dict(m=np.ones(r["n"]), L=r["L"])) for r in reps]
    x, v = _t(np.concatenate([r["pos"] for r in reps])), _t(np.concatenate([r["vel"] for r in reps]))
    atom = torch.cat([torch.arange(r["n"], device=DEVICE) for r in reps])
    key = torch.cat([torch.full((r["n"],), 1000 + k, device=DEVICE) for k, r in enumerate(reps)])
    sd = torch.cat([torch.full((r["n"], 1), math.sqrt((1 - c1 * c1) * r["T"]), dtype=torch.float64, device=DEVICE) for r in reps])

    def accel(x):
        return torch.cat([e.accel(x[i:j]) for e, i, j in zip(forces, ends[:-1], ends[1:])])

    a = accel(x)
    for k in range(case["steps"]):
        v = v + 0.5 * dt * a
        x = x + 0.5 * dt * v
        v = c1 * v + sd * _normals(key, atom, k)
        x = x + 0.5 * dt * v
        a = accel(x)
        v = v + 0.5 * dt * a
    return {"u": x.cpu().numpy(), "v": v.cpu().numpy()}


def _exact_rdf(case, seed):
    frames, L = _frames(case, seed)
    dr = L / case["maxbin"]
    hist = torch.zeros(case["maxbin"], dtype=torch.int64, device=DEVICE)
    n = case["n_mol"]
    later = torch.triu(torch.ones(n, n, dtype=torch.bool, device=DEVICE), 1)
    for frame in frames:
        x = _t(frame[::3])
        d = x[:, None, :] - x[None, :, :]
        d = d - L * torch.round(d / L)
        r2 = (d[..., 0] ** 2 + d[..., 1] ** 2) + d[..., 2] ** 2
        bins = torch.ceil(torch.sqrt(r2) / dr).long()[later & (r2 < (0.5 * L) ** 2)]
        hist += 2 * torch.bincount(bins[(bins >= 2) & (bins <= case["maxbin"])] - 1, minlength=case["maxbin"])
    return hist.double().cpu().numpy()


def _exact_gradient(case, seed):
    theta, x, y = (_t(a) for a in _gradient_inputs(case, seed))
    sizes = [ND * NH, NH, NH * NH, NH, NH, 1]
    w1, b1, w2, b2, w3, b3 = torch.split(theta[:sum(sizes)], sizes)
    w1, w2 = w1.view(ND, NH), w2.view(NH, NH)
    a1 = torch.tanh(x @ w1 + b1)
    a2 = torch.tanh(a1 @ w2 + b2)
    err = a2 @ w3 + b3 - y
    de = 2 * err / len(y)
    g2 = de[:, None] * w3 * (1 - a2 * a2)
    g1 = (g2 @ w2.T) * (1 - a1 * a1)
    grad = torch.cat([(x.T @ g1).reshape(-1), g1.sum(0), (a1.T @ g2).reshape(-1), g2.sum(0), a2.T @ de, de.sum().view(1)])
    return {"loss": float((err * err).mean()), "grad": grad.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "rdf":
        return _exact_rdf(case, seed)
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if case["system"] == "batch":
        n = case["replicas"] * (0.5 * (case["n_min"] + case["n_max"])) ** 2
        return _exact_batch(case, seed) if n * case["steps"] < 1.5e11 else None
    s = _inputs(case, seed)
    e = _Exact(case, s)
    if kind == "energy":
        out = e.energies(_t(s["u"]), _t(s["v"]))
        out["temperature"] = 2 * out["kinetic"] / (s["kb"] * e.ndf())
        return out
    if kind == "rhs":
        x, v = _t(s["u"]), _t(s["v"])
        a = e.accel(x)
        T = float((e.m[:, None] * v * v).sum()) / (s["kb"] * e.ndf())
        if case["thermostat"] == "berendsen":
            a = a + 0.5 / 0.1 * (s["T0"] / T - 1.0) * v
        a = a.cpu().numpy()
        return np.concatenate([a, np.zeros((1, 3))]) if case["thermostat"] == "nosehoover" else a
    if float(e.n) ** 2 * case["steps"] > 1.5e11:
        return None  # minutes of 64-bit all-pairs work
    return _exact_run(case, s)
