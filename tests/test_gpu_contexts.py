"""Contexts of different sizes in one process: what a later, smaller one needs
takes nothing away from an earlier, larger one."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _batch(sizes):
    descs, keep, us, vs = [], [], [], []
    for r, n in enumerate(sizes):
        pos, vel, L = nbg.workloads.lj_argon_lattice(n, seed=r, jitter=0.05)
        d, k = nbg.lennard_jones_descriptor(np.ones(n), L, seed=r, skin=0.3, thermostat=nbg.LangevinThermostat(1.0, 1.0))
        d.flags |= nbg._abi.NBG_FLAG_LANGEVIN_BAOAB
        descs.append(d)
        keep.append(k)
        us.append(pos)
        vs.append(vel)
    return descs, keep, np.concatenate(us), np.concatenate(vs)


def test_smaller_batch_after_a_larger_one(gpu):
    descs, keep, u, v = _batch([8000, 300])
    large = nbg.Engine(descs, 0)
    assert large.ensemble_form() is not None
    want = large.run(u, v, 0.004, 5, 0, save_trajectory=False, step=0)
    descs2, keep2, u2, v2 = _batch([300, 150])
    small = nbg.Engine(descs2, 0)
    assert small.ensemble_form() is not None
    small.run(u2, v2, 0.004, 5, 0, save_trajectory=False, step=0)
    got = large.run(u, v, 0.004, 5, 0, save_trajectory=False, step=0)
    for k in range(2):
        np.testing.assert_array_equal(got[k], want[k])
    small.close()
    large.close()


def _forces(eng, u, v):
    eng.set_state(u, v)
    eng.compute_forces()
    return eng.get_accel()


# the per-block staging form: its shared memory follows the row capacity
@pytest.mark.parametrize("lanes", [16, 32])
def test_shorter_rows_after_longer_ones(gpu, oracle, monkeypatch, lanes):
    monkeypatch.setenv("NBG_FX_BLOCK", "1")
    monkeypatch.setenv("NBG_LIST_LPA", str(lanes))
    monkeypatch.setenv("NBG_NO_CLUSTER", "1")
    sim = S.water_box(1000, seed=6)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    water = nbg.Engine(desc, 0)
    assert water.force_form() == (lanes, True)
    a = _forces(water, u, v)
    sim2 = S.water_box(1000, seed=6, R=0.5)
    desc2, keep2 = nbg.system_descriptor(sim2)
    other = nbg.Engine(desc2, 0)
    assert other.force_form() == (lanes, True)
    assert S.rel_rmse(_forces(other, u, v), oracle.accel(desc2, v.copy(), u)[0]) <= 1e-5
    np.testing.assert_array_equal(_forces(water, u, v), a)
    assert S.rel_rmse(a, oracle.accel(desc, v.copy(), u)[0]) <= 1e-5
    other.close()
    water.close()
