"""The right-hand side off the Verlet lists through the pinned staging (up to
16,384 columns; a Nose-Hoover system has one more than bodies): thermostat
terms against the oracle, repeated calls, and the bodies on both sides of the
line against a direct FP64 sum."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # FP32 pair arithmetic, as everywhere


def _ions(n, thermostat=()):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    g = np.arange(side) + 0.5
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n] + rng.uniform(-0.2, 0.2, (n, 3))
    v = rng.standard_normal((n, 3))
    q = rng.choice([-1.0, 1.0], n)
    bodies = [nbg.ChargedParticle(x[i], v[i], 1.0, q[i]) for i in range(n)]
    system = nbg.PotentialNBodySystem(bodies, {"electrostatic": nbg.ElectrostaticParameters(1.5)})
    return nbg.NBodySimulation(system, (0.0, 1.0), *thermostat, kb=1.0), x, q


@pytest.mark.parametrize("thermostat", ["none", "berendsen", "nosehoover"])
@pytest.mark.parametrize("n", [2, 257])
def test_staged_rhs_thermostats(gpu, oracle, n, thermostat):
    th = {"none": [], "berendsen": [nbg.BerendsenThermostat(0.9, 0.1)], "nosehoover": [nbg.NoseHooverThermostat(0.9, 0.5)]}
    sim, _, _ = _ions(n, th[thermostat])
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    for k in range(3):
        w = v * (1.0 + 0.1 * k)
        wo = w.copy()
        a = eng.accel(w, u)
        ar, vo = oracle.accel(desc, wo, u)
        assert S.rel_rmse(a[:n], ar[:n]) <= FORCE_TOL
        assert np.isfinite(w).all()
        u = u + 0.01
    eng.close()


@pytest.mark.parametrize("n", [16384, 16385])
def test_staged_rhs_line(gpu, n):
    sim, x, q = _ions(n)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    a = eng.accel(v.copy(), u)
    eng.close()
    pick = np.r_[0, n - 1, np.random.default_rng(1).integers(0, n, 20)]
    ref = np.empty((len(pick), 3))
    for k, i in enumerate(pick):
        d = x[i] - x
        r2 = (d * d).sum(1)
        r2[i] = np.inf
        ref[k] = (1.5 * q[i] * q / r2**1.5) @ d
    assert S.rel_rmse(a[pick], ref) <= FORCE_TOL
