"""Runs whose Verlet lists overflow on the first evaluation (a dense droplet in
a wide box): after the lists have grown, the first steps start from the
acceleration of the whole pair set, on every step loop, in nbg_run and in a
deferred nbg_advance, against the FP64 oracle."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

DT = 0.001


def _droplet(side, L, seed=0, thermostat=None):
    """A cubic droplet of density about 1 and the descriptor of its box."""
    n = side**3
    rng = np.random.default_rng(seed)
    g = np.arange(side) * 1.0 + 5.0
    u = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.02, 0.02, (n, 3))
    d, keep = nbg.lennard_jones_descriptor(np.ones(n), L, skin=0.5, seed=seed + 3, thermostat=thermostat)
    return d, keep, u, rng.standard_normal((n, 3))


def _check(d, u, v, u1, v1, ur, vr):
    """FP32 forces, 1e-6 of the largest, over a few steps: positions to 1e-6 of the box, velocities to 1e-5 of the
    fastest atom."""
    assert np.abs(u1 - ur).max() <= 1e-6 * d.box[0]
    assert np.abs(v1 - vr).max() <= 1e-5 * np.abs(vr).max()


# the small-system loop; the same on step graphs and single steps; a larger system
@pytest.mark.parametrize("side,L,env", [(7, 24.0, {}), (7, 24.0, {"NBG_NO_CLUSTER": "1"}),
                                        (7, 24.0, {"NBG_NO_CLUSTER": "1", "NBG_LIST_LPA": "1"}), (14, 45.0, {})])
@pytest.mark.parametrize("steps", [1, 3, 20])
def test_first_steps_after_regrowth(gpu, oracle, monkeypatch, side, L, env, steps):
    for k, x in env.items():
        monkeypatch.setenv(k, x)
    d, keep, u, v = _droplet(side, L)
    ur, vr = oracle.run(d, u, v, DT, steps)
    eng = nbg.Engine(d, 0)
    assert eng.force_form() is not None
    u1, v1, _, _, _ = eng.run(u, v, DT, steps, 0, save_trajectory=False)
    eng.close()
    _check(d, u, v, u1, v1, ur, vr)
    eng = nbg.Engine(d, 0)
    eng.set_state(u, v)
    eng.advance(DT, steps)
    u2, v2 = eng.get_state()
    eng.close()
    _check(d, u, v, u2, v2, ur, vr)


@pytest.mark.parametrize("how", ["run", "advance", "tune", "graphs"])
def test_first_steps_of_a_batch_after_regrowth(gpu, oracle, monkeypatch, how):
    if how == "graphs":
        monkeypatch.setenv("NBG_NO_ENSEMBLE_LOOP", "1")
    reps = [_droplet(side, 24.0, seed=r, thermostat=nbg.LangevinThermostat(0.7, 1.0)) for r, side in enumerate((5, 6, 7))]
    for r in reps:
        r[0].flags |= nbg._abi.NBG_FLAG_LANGEVIN_BAOAB
    u, v = np.concatenate([r[2] for r in reps]), np.concatenate([r[3] for r in reps])
    eng = nbg.Engine([r[0] for r in reps], 0)
    if how == "tune":
        eng.set_state(u, v)
        eng.ensemble_tune(2)
    if how in ("run", "graphs"):
        u1, v1, _, _, _ = eng.run(u, v, DT, 3, 0, save_trajectory=False, step=0)
    else:
        if how == "advance":
            eng.set_state(u, v)
        eng.set_step(0)
        eng.advance(DT, 3)
        u1, v1 = eng.get_state()
    eng.close()
    off = 0
    for d, _, ui, vi in reps:
        s = slice(off, off + int(d.n))
        _check(d, ui, vi, u1[s], v1[s], *oracle.run(d, ui, vi, DT, 3))
        off += int(d.n)


# the chunk that overflowed has moved the thermostat's column too
@pytest.mark.parametrize("steps", [1, 5, 40])
def test_nosehoover_column_after_regrowth(gpu, oracle, steps):
    d, keep, u, v = _droplet(14, 45.0, thermostat=nbg.NoseHooverThermostat(0.7, 0.05))
    u, v = np.concatenate([u, np.zeros((1, 3))]), np.concatenate([v, np.zeros((1, 3))])
    ur, vr = oracle.run(d, u, v, DT, steps)
    eng = nbg.Engine(d, 0)
    u1, v1, _, _, _ = eng.run(u, v, DT, steps, 0, save_trajectory=False)
    eng.close()
    _check(d, u, v, u1[:-1], v1[:-1], ur[:-1], vr[:-1])
    assert abs(u1[-1, 0] - ur[-1, 0]) <= 1e-5 * abs(ur[-1, 0])
    assert abs(v1[-1, 0] - vr[-1, 0]) <= 1e-5 * abs(vr[-1, 0])
