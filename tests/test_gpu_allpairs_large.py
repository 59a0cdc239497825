"""The all-pairs forms beyond their small-system shapes: more tiles per CTA than
it has warps (from 8193 bodies on), and the line to the general kernel (256
tiles, 32,768 bodies), against a direct FP64 sum of a sample of bodies."""
import math

import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _system(form, n):
    rng = np.random.default_rng(n)
    side = math.ceil(n ** (1 / 3))
    L = 1.1 * side
    g = (np.arange(side) + 0.5) * L / side
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n] + rng.uniform(-0.1, 0.1, (n, 3))
    m, q = rng.uniform(0.5, 1.5, n), rng.choice([-1.0, 1.0], n)
    cubic = form.endswith("cubic")
    lj = nbg.LennardJonesParameters(1.0, 1.0, 3.0 if cubic else 2.5)
    pots = {"lennard_jones": lj}
    Rel = math.inf
    if "coulomb" in form:
        Rel = 0.45 * L if cubic else math.inf
        pots["electrostatic"] = nbg.ElectrostaticParameters(1.5, Rel) if cubic else nbg.ElectrostaticParameters(1.5)
    bodies = [nbg.ChargedParticle(*b) for b in zip(x, np.zeros((n, 3)), m, q)]
    bc = [nbg.CubicPeriodicBoundaryConditions(L)] if cubic else []
    sim = nbg.NBodySimulation(nbg.PotentialNBodySystem(bodies, pots), (0.0, 1.0), *bc, kb=1.0,
                              flags=nbg._abi.NBG_FLAG_ALL_PAIRS)

    def accel(i):
        d = x[i] - x
        if cubic:
            d -= L * np.round(d / L)
        r2 = (d * d).sum(axis=1)
        r2[i] = np.inf
        s6 = 1.0 / r2**3
        f = np.where(r2 < lj.R**2, 24.0 * (2.0 * s6 * s6 - s6) / r2, 0.0)
        if "coulomb" in form:
            f = f + np.where(r2 < Rel**2, 1.5 * q[i] * q / r2**1.5, 0.0)
        return f @ d / m[i]

    return sim, accel


@pytest.mark.parametrize("form,n", [(f, n) for f in ("lj-cubic", "lj-coulomb-cubic", "lj-coulomb") for n in (8192, 8193)]
                         + [("lj-coulomb-cubic", n) for n in (12345, 32768, 32769)])
def test_allpairs_sample(gpu, form, n):
    sim, accel = _system(form, n)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is None  # off the lists
    a = eng.accel(v.copy(), u)
    eng.close()
    pick = np.r_[0, 127, 128, n - 1, np.random.default_rng(1).integers(0, n, 40)]
    ref = np.stack([accel(i) for i in pick])
    assert S.rel_rmse(a[pick], ref) <= 1e-5  # FP32 pair arithmetic, as everywhere
