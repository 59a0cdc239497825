"""Positions that are not finite, off the Verlet lists: the right-hand side and
a run end with NBG_ERR_NONFINITE on every form of the all-pairs kernel, the
context stays usable, and a finite position out of FP32's range for r^2 is
accepted (it interacts with nobody)."""
import math

import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

NONFINITE = -4


def _system(form, n):
    rng = np.random.default_rng(n)
    side = math.ceil(n ** (1 / 3))
    L = 1.1 * side
    g = (np.arange(side) + 0.5) * L / side
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n] + rng.uniform(-0.1, 0.1, (n, 3))
    v, m, q = np.zeros((n, 3)), rng.uniform(0.5, 1.5, n), rng.choice([-1.0, 1.0], n)
    if form == "water":
        return S.water_box(n // 3, seed=n, R=0.45 * (n / 3 / 33.3) ** (1 / 3))
    lj, el = nbg.LennardJonesParameters(1.0, 1.0, 0.4 * L), nbg.ElectrostaticParameters(1.5)
    pots = {"coulomb": {"electrostatic": el}, "lj-open": {"lennard_jones": nbg.LennardJonesParameters(1.0, 1.0, math.inf)},
            "lj-cubic": {"lennard_jones": lj}, "lj-coulomb": {"lennard_jones": lj, "electrostatic": el},
            "lj-coulomb-cubic": {"lennard_jones": lj, "electrostatic": nbg.ElectrostaticParameters(1.5, 0.45 * L)},
            "lj-gravity": {"lennard_jones": lj, "gravitational": nbg.GravitationalParameters(1.0)}}[form]
    bc = [nbg.CubicPeriodicBoundaryConditions(L)] if form.endswith("cubic") else []
    bodies = [nbg.ChargedParticle(*b) for b in zip(x, v, m, q)]
    return nbg.NBodySimulation(nbg.PotentialNBodySystem(bodies, pots), (0.0, 1.0), *bc, kb=1.0,
                               flags=nbg._abi.NBG_FLAG_ALL_PAIRS)


# a tile per CTA up to 2048 bodies, then a tile per warp; the body in the
# first tile, in the last one, and alone in its own
@pytest.mark.parametrize("n,bad", [(2, 1), (200, 3), (129, 128), (2500, 7), (2500, 2499)])
@pytest.mark.parametrize("form", ["coulomb", "lj-open", "lj-cubic", "lj-coulomb", "lj-coulomb-cubic", "lj-gravity"])
def test_nonfinite_position_is_reported(gpu, form, n, bad):
    sim = _system(form, n)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    good = eng.accel(v.copy(), u)
    for value in (np.nan, -np.nan, np.inf, -np.inf):
        w = u.copy()
        w[bad, 1] = value
        for call in (lambda: eng.accel(v.copy(), w), lambda: eng.run(w, v, 1e-3, 3, 0, save_trajectory=False),
                     lambda: eng.run(w, v, 1e-3, 20, 0, save_trajectory=False)):
            with pytest.raises(nbg.EngineError) as ei:
                call()
            assert ei.value.status == NONFINITE
        np.testing.assert_array_equal(eng.accel(v.copy(), u), good)
    eng.close()


def test_nonfinite_position_is_reported_for_water(gpu):
    sim = _system("water", 192)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is None  # off the lists
    u[9, 2] = np.nan
    with pytest.raises(nbg.EngineError) as ei:
        eng.accel(v.copy(), u)
    assert ei.value.status == NONFINITE
    eng.close()


@pytest.mark.parametrize("n", [200, 2500])
@pytest.mark.parametrize("form", ["coulomb", "lj-open", "lj-coulomb"])
def test_far_position_interacts_with_nobody(gpu, oracle, form, n):
    sim = _system(form, n)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    u[5] = [1e25, -1e25, 1e25]
    eng = nbg.Engine(desc, 0)
    a = eng.accel(v.copy(), u)
    eng.close()
    ref, _ = oracle.accel(desc, v, u)
    assert not a[5].any()
    assert S.rel_rmse(a, ref) <= 1e-5  # FP32 pair arithmetic, as everywhere
