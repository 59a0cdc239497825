"""The persistent cluster loop of small systems by potential (Lennard-Jones,
electrostatic, both) at the edges of its shapes (atoms per CTA, lanes per atom,
CTAs without atoms): accelerations against the oracle, and a run with saved
frames against the step graphs."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # FP32 pair arithmetic, as everywhere


def _sim(n, pots):
    pos, vel, L = nbg.workloads.lj_argon_lattice(n, seed=n, jitter=0.05)
    R = min(2.5, 0.42 * L)
    q = np.random.default_rng(n).choice([-1.0, 1.0], n)
    bodies = [nbg.ChargedParticle(pos[i], vel[i], 1.0, q[i]) for i in range(n)]
    p = {}
    if "lj" in pots:
        p["lennard_jones"] = nbg.LennardJonesParameters(1.0, 1.0, R)
    if "el" in pots:
        p["electrostatic"] = nbg.ElectrostaticParameters(1.5, 0.9 * R, eps_rf=1.0)
    system = nbg.PotentialNBodySystem(bodies, p)
    return nbg.NBodySimulation(system, (0.0, 1.0), nbg.CubicPeriodicBoundaryConditions(L), kb=1.0, skin=0.3, seed=5)


@pytest.mark.parametrize("pots", ["lj", "el", "lj+el"])
@pytest.mark.parametrize("n", [64, 65, 145, 512, 513, 1024, 1025, 1700])
def test_cluster_loop(gpu, oracle, monkeypatch, n, pots):
    sim = _sim(n, pots)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    dt, steps = 1e-3, 31
    eng = nbg.Engine(desc, 0)
    a = eng.accel(v.copy(), u)
    ar, _ = oracle.accel(desc, v, u)
    assert S.rel_rmse(a, ar) <= FORCE_TOL
    got = eng.run(u, v, dt, steps, save_every=3, step=2)
    eng.close()
    monkeypatch.setenv("NBG_NO_CLUSTER", "1")
    ref = nbg.Engine(desc, 0)
    want = ref.run(u, v, dt, steps, save_every=3, step=2)
    ref.close()
    # two FP32 force forms, each within 1e-5 of the largest acceleration:
    # the velocities part by t da, the positions by t^2 da / 2
    t, da = steps * dt, 2 * FORCE_TOL * np.abs(ar).max()
    for k, tol in ((0, t * t * da), (1, 2 * t * da), (2, t * t * da), (3, 2 * t * da)):
        x, y = np.asarray(got[k]), np.asarray(want[k])
        assert x.shape == y.shape
        assert np.abs(x - y).max() <= tol, k
