"""The all-pairs kernel at the edges of its 32-body blocks, 128-body tiles and
rounds of 16 tiles (10 in its general form), against the FP64 oracle."""
import math

import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _system(form, n):
    rng = np.random.default_rng(n)
    side = math.ceil(n ** (1 / 3))
    L = 1.1 * max(side, 2)
    g = (np.arange(side) + 0.5) * L / side
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n] + rng.uniform(-0.1, 0.1, (n, 3))
    v, m, q, mm = np.zeros((n, 3)), rng.uniform(0.5, 1.5, n), rng.choice([-1.0, 1.0], n), rng.standard_normal((n, 3))
    cubic = [nbg.CubicPeriodicBoundaryConditions(L)]
    lj = nbg.LennardJonesParameters(1.0, 1.0, 0.49 * L)
    if form == "lj-cubic":
        bodies, pots, bc = [nbg.MassBody(*b) for b in zip(x, v, m)], {"lennard_jones": lj}, cubic
    elif form == "coulomb":
        bodies, pots, bc = [nbg.ChargedParticle(*b) for b in zip(x, v, m, q)], \
            {"electrostatic": nbg.ElectrostaticParameters(1.5)}, []
    elif form == "lj-coulomb-cubic":
        bodies, pots, bc = [nbg.ChargedParticle(*b) for b in zip(x, v, m, q)], \
            {"lennard_jones": lj, "electrostatic": nbg.ElectrostaticParameters(1.5, 0.45 * L)}, cubic
    elif form == "lj-gravity":
        bodies, pots, bc = [nbg.MassBody(*b) for b in zip(x, v, m)], \
            {"lennard_jones": lj, "gravitational": nbg.GravitationalParameters(1.0)}, []
    else:
        bodies, pots, bc = [nbg.MagneticParticle(*b) for b in zip(x, v, m, mm)], \
            {"magnetostatic": nbg.MagnetostaticParameters(1.0)}, []
    return nbg.NBodySimulation(nbg.PotentialNBodySystem(bodies, pots), (0.0, 1.0), *bc, kb=1.0,
                               flags=nbg._abi.NBG_FLAG_ALL_PAIRS)


# FP32 pair terms (a few 2^-24 each) summed over at most 128 in FP32 and
# compensated beyond; dipole and alternating-charge sums cancel by up to ~1e2
@pytest.mark.parametrize("n", [2, 31, 33, 127, 129, 1281, 2047, 2049])
@pytest.mark.parametrize("form", ["lj-cubic", "coulomb", "lj-coulomb-cubic", "lj-gravity", "dipoles"])
def test_allpairs_tile_edges(gpu, oracle, form, n):
    sim = _system(form, n)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    a = eng.accel(v.copy(), u)
    ref, _ = oracle.accel(desc, v, u)
    assert np.linalg.norm(a - ref) <= 1e-5 * np.linalg.norm(ref)
    eng.close()
