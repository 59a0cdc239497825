"""The fused step kernels of the captured step graphs (kick, thermostat,
Andersen collisions, saved frame and next drift in one launch) against single
steps launched one by one (NBG_NO_GRAPHS): the same bits, frames included, at
run lengths that are not a whole number of graphs."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _sim(system, thermostat):
    T = 300.0 if system.startswith("water") else 0.9
    th = {"none": [], "berendsen": [nbg.BerendsenThermostat(T, 0.1)], "nosehoover": [nbg.NoseHooverThermostat(T, 0.5)],
          "andersen": [nbg.AndersenThermostat(T, 3.0)]}[thermostat]
    if system.startswith("water"):
        return S.water_box({"water-list": 950, "water-pairs": 11}[system], seed=3, thermostat=th[0] if th else None)
    if system == "gravity":
        pos, vel, m = nbg.workloads.plummer_sphere(333, seed=1)
        m = m * np.random.default_rng(1).uniform(0.5, 1.5, len(m))
        bodies = [nbg.MassBody(*b) for b in zip(pos, vel, m)]
        return nbg.NBodySimulation(nbg.GravitationalSystem(bodies, 1.0), (0.0, 1.0), *th, kb=1.0)
    n = {"lj-list": 2531, "lj-pairs": 131}[system]
    pos, vel, L = nbg.workloads.lj_argon_lattice(n, seed=2, jitter=0.05)
    bodies = [nbg.MassBody(*b) for b in zip(pos, vel, np.ones(n))]
    lj = nbg.PotentialNBodySystem(bodies, {"lennard_jones": nbg.LennardJonesParameters(1.0, 1.0, 2.5)})
    return nbg.NBodySimulation(lj, (0.0, 1.0), nbg.CubicPeriodicBoundaryConditions(L), *th, kb=1.0, skin=0.3, seed=5)


@pytest.mark.parametrize("thermostat", ["none", "berendsen", "nosehoover", "andersen"])
@pytest.mark.parametrize("system", ["lj-list", "lj-pairs", "water-list", "water-pairs", "gravity"])
def test_fused_steps_match_single_steps(gpu, monkeypatch, system, thermostat):
    sim = _sim(system, thermostat)
    u, v = S.state(sim)
    dt = 5e-4 if system.startswith("water") else 2e-3
    out = []
    for graphs in (True, False):
        if not graphs:
            monkeypatch.setenv("NBG_NO_GRAPHS", "1")
        desc, keep = nbg.system_descriptor(sim)
        eng = nbg.Engine(desc, 0)
        a = eng.run(u, v, dt, 37, save_every=3, step=0)
        b = eng.run(a[0], a[1], dt, 40, save_every=0)
        out.append([*a[:4], b[0], b[1]])
        eng.close()
    for x, y in zip(*out):
        np.testing.assert_array_equal(x, y)
