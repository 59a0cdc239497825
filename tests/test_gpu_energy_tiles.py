"""The energy kernels at the edges of their 128 x 32 items (all pairs) and of
their queues (lists), and on positions many boxes out, against the FP64
oracle. Sums of n FP64 terms: 1e-11 of the largest partial sum's scale."""
import math

import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _box(n):
    rng = np.random.default_rng(n)
    side = math.ceil(n ** (1 / 3))
    L = 1.1 * max(side, 2)
    g = (np.arange(side) + 0.5) * L / side
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n] + rng.uniform(-0.1, 0.1, (n, 3))
    return x, rng.standard_normal((n, 3)), rng.uniform(0.5, 1.5, n), rng.choice([-1.0, 1.0], n), L, rng


def _lj_energy(x, L, R=2.5):
    """4 sum_{i<j} (s^12 - s^6), r clamped to R, eps = sigma = 1, to rounding: numpy's pairwise sums of each row,
    math.fsum over the rows. (The oracle adds the 12.5 million terms of 5001 atoms one after the other, which
    rounds its sum by 2e-10.)"""
    rows = []
    for i in range(len(x) - 1):
        d = x[i] - x[i + 1:]
        d -= L * np.round(d / L)
        s6 = (1.0 / np.minimum((d * d).sum(axis=1), R * R)) ** 3
        rows.append(float((s6 * s6 - s6).sum()))
    return 4.0 * math.fsum(rows)


def _check(gpu_e, ref):
    for k, r in ref.items():
        assert abs(gpu_e[k] - r) <= 1e-11 * (abs(r) + abs(ref["kinetic"])), k


@pytest.mark.parametrize("n", [2, 31, 33, 127, 128, 129, 700])
@pytest.mark.parametrize("form", ["coulomb", "lj-cubic", "lj-coulomb-periodic", "gravity"])
def test_pair_energies(gpu, oracle, form, n):
    x, v, m, q, L, rng = _box(n)
    lj = nbg.LennardJonesParameters(1.0, 1.0, 0.45 * L)
    bc = []
    if form == "coulomb":
        sysm = nbg.ChargedParticles([nbg.ChargedParticle(*b) for b in zip(x, v, m, q)], 1.5)
    elif form == "gravity":
        sysm = nbg.GravitationalSystem([nbg.MassBody(*b) for b in zip(x, v, m)], 1.0)
    elif form == "lj-cubic":
        x = x + L * rng.integers(-3, 4, (n, 3))  # unwrapped positions
        sysm = nbg.PotentialNBodySystem([nbg.MassBody(*b) for b in zip(x, v, m)], {"lennard_jones": lj})
        bc = [nbg.CubicPeriodicBoundaryConditions(L)]
    else:
        sysm = nbg.PotentialNBodySystem([nbg.ChargedParticle(*b) for b in zip(x, v, m, q)],
                                        {"lennard_jones": lj, "electrostatic": nbg.ElectrostaticParameters(1.5, 0.4 * L)})
        bc = [nbg.PeriodicBoundaryConditions([-0.5 * L, 0.5 * L] * 3)]
    sim = nbg.NBodySimulation(sysm, (0.0, 1.0), *bc, kb=1.0, flags=nbg._abi.NBG_FLAG_ALL_PAIRS)
    desc, keep = nbg.system_descriptor(sim)
    u, vel = S.state(sim)
    eng = nbg.Engine(desc, 0)
    _check(eng.energy(u, vel), oracle.energy(desc, u, vel))
    eng.close()


@pytest.mark.parametrize("shift", [0, 5])
@pytest.mark.parametrize("kind,size", [("lj", 600), ("lj", 5001), ("water", 950)])
def test_list_energies(gpu, oracle, kind, size, shift):
    if kind == "lj":
        u, v, L = nbg.workloads.lj_argon_lattice(size, rho=0.8, seed=size, jitter=0.1)
        desc, keep = nbg.lennard_jones_descriptor(np.ones(size), L)
    else:
        sim = S.water_box(size, seed=size)
        desc, keep = nbg.system_descriptor(sim)
        u, v = S.state(sim)
        L = desc.box[0]
    # whole molecules (or atoms) several boxes out, as after a long run
    per = 3 if kind == "water" else 1
    u = u + L * np.repeat(np.random.default_rng(1).integers(-shift, shift + 1, (len(u) // per, 3)), per, axis=0)
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is not None
    ref = oracle.energy(desc, u, v)
    if kind == "lj":
        ref["lennard_jones"] = ref["potential"] = _lj_energy(u, L)
        ref["total"] = ref["kinetic"] + ref["potential"]
    _check(eng.energy(u, v), ref)
    eng.close()
