"""Energies of states with a lost atom. A NaN coordinate of either sign counts
as beyond every cutoff (no comparison with it holds), in both energy kernels."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["pairs", "list-split", "list-hi"])
def test_nan_position_of_either_sign(gpu, system):
    n = {"pairs": 300, "list-split": 3000, "list-hi": 12000}[system]
    u, v, L = nbg.workloads.lj_argon_lattice(n, seed=n, jitter=0.1)
    desc, keep = nbg.lennard_jones_descriptor(np.ones(n), L)
    if system == "pairs":
        desc.flags |= nbg._abi.NBG_FLAG_ALL_PAIRS
    eng = nbg.Engine(desc, 0)
    whole = eng.energy(u, v)
    got = []
    for value in (np.nan, -np.nan):
        w = u.copy()
        w[17, 1] = value
        got.append(eng.energy(w, v))
    eng.close()
    assert got[0] == got[1]
    d = u[17] - np.delete(u, 17, axis=0)
    d -= L * np.round(d / L)
    r2 = (d * d).sum(axis=1)
    s6 = (1.0 / np.minimum(r2, 2.5**2)) ** 3  # the atom's pairs, and the same at the cutoff
    cut = 2.5**-6
    lost = 4.0 * ((s6 * s6 - s6).sum() - (n - 1) * (cut * cut - cut))
    assert abs(got[0]["lennard_jones"] - (whole["lennard_jones"] - lost)) <= 1e-11 * abs(whole["lennard_jones"])
